"""The checkpointed forward of the adjoint is a recursion of one moment set with FP64 products, so every form
of the step can be asked for, and gives the moments of the others up to the order of their sums: at most
4 n 2^-53 ||v|| ||T_m v|| apart, ||T_m v|| <= ||v|| for a Hermitian operator within its bounds (and 2^-40 of
that for the rounding that M orders of a recursion add up)."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 2, 4])
@pytest.mark.parametrize("nx,ny", [(9, 7), (150, 131)])
def test_every_form_serves_the_forward(cuda_lib, nx, ny, R):
    import torch

    from minijclsquant_gb300 import device, lattice

    g = lattice.honeycomb_device(nx, ny, W=1.0, seed=2)
    th = torch.from_numpy(np.random.default_rng(3).uniform(0, 6.28, (R, g.n))).cuda()
    v = torch.polar(torch.ones_like(th), th)
    M, want = 30, None
    forms = {"simple": (0, 1), "staged1": (1, 1), "staged2": (1, 2), "ws1": (2, 1), "ws2": (2, 2)}
    for form, expect in forms.items():
        os.environ["KPM_STEP_KERNEL"] = form
        try:
            op = device.DeviceELL(g.data_kpm, g.indices, g.len_row)
            kind, U = ctypes.c_int(), ctypes.c_int()
            assert cuda_lib.kpm_adjoint_step_config(op.handle, R, ctypes.byref(kind), ctypes.byref(U), None, None) == 0
            assert (kind.value, U.value) == expect, form
            mu = torch.empty((R, M), dtype=torch.complex128, device="cuda")
            assert cuda_lib.kpm_adjoint_forward(op.handle, R, M, 8, v.data_ptr(), mu.data_ptr(),
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            assert cuda_lib.kpm_ell_check(op.handle, None) == 0
        finally:
            del os.environ["KPM_STEP_KERNEL"]
        want = mu if want is None else want
        assert torch.max((mu - want).abs()).item() <= (4 * g.n * 2.0 ** -53 + 2.0 ** -40) * g.n
    assert cuda_lib.kpm_adjoint_step_config(None, 1, None, None, None, None) != 0
    assert cuda_lib.kpm_adjoint_step_config(op.handle, 3, None, None, None, None) != 0
