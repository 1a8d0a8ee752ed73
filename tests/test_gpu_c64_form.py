"""complex64 moments of operators that are not large take their step form by size: the same form and the
same bits for a new handle of the shape, and the moments of the complex128 recursion to the complex64
tolerance of the step-kernel tests (2e-6 of the number of sites)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(210, 200), (335, 300), (400, 380)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("R", [1, 2, 4, 8])
def test_form_by_size(cuda_lib, nx, ny, cplx, R):
    import torch

    from minijclsquant_gb300 import _capi, device, lattice

    g = lattice.honeycomb_device(nx, ny, W=1.0, seed=1)
    n, L = g.n, g.len_row
    data = g.data_kpm
    if cplx:  # a gauge: complex values, the same spectrum
        th = torch.from_numpy(np.random.default_rng(2).uniform(0, 6.28, n)).cuda()
        ix = g.indices.view(n, L).long()
        ph = torch.polar(torch.ones((n, L), dtype=torch.float64, device="cuda"), th[:, None] - th[ix])
        data = (data.view(n, L) * ph).reshape(-1).contiguous()
    th = torch.from_numpy(np.random.default_rng(3).uniform(0, 6.28, (R, n))).cuda()
    v = torch.polar(torch.ones_like(th), th)
    seen = []
    for _ in range(2):
        op = device.DeviceELL(data, g.indices, L)
        c = [ctypes.c_int() for _ in range(3)]
        assert cuda_lib.kpm_ell_step_config(op.handle, _capi.KPM_C64, R, *map(ctypes.byref, c), None) == 0
        mu = device.cheb_moments(op, 60, v, dtype="c64").cpu().numpy()
        assert cuda_lib.kpm_ell_check(op.handle, None) == 0
        seen.append(([x.value for x in c], mu))
    assert seen[0][0] == seen[1][0] and seen[0][0][0] == (1 if cplx and R == 2 and n < 200000 else 2)
    assert np.array_equal(seen[0][1], seen[1][1])
    ref = device.cheb_moments(op, 60, v).cpu().numpy()
    assert np.max(np.abs(seen[0][1] - ref)) <= 2e-6 * n
