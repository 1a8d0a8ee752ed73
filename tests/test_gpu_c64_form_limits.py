"""The complex64 step forms by size on both sides of every limit, whichever operator of the same padded size
came first in the process, and the moments of the forms beyond 304,000 sites (test_gpu_c64_form has those
below) within the complex64 tolerance of the step-kernel tests (2e-6 of the number of sites)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (complex, R, n) -> (kind, rows per thread)
LIMITS = [(False, 1, 720000, 2, 2), (False, 1, 720001, 2, 1), (False, 2, 299999, 2, 2), (False, 2, 300000, 2, 1),
          (False, 4, 299999, 2, 2), (False, 4, 300000, 2, 1), (False, 8, 199999, 2, 2), (False, 8, 799999, 2, 2),
          (True, 1, 199999, 2, 2), (True, 1, 200000, 2, 1), (True, 1, 599999, 2, 1), (True, 1, 600000, 0, 1),
          (True, 2, 199999, 1, 2), (True, 2, 200000, 2, 1), (True, 4, 114999, 2, 2), (True, 4, 115000, 2, 1),
          (True, 8, 100000, 2, 1), (True, 8, 799999, 2, 1)]


def _config(lib, n, R, cplx):
    import torch

    from minijclsquant_gb300 import _capi
    from minijclsquant_gb300.device import DeviceELL

    op = DeviceELL(torch.full((n,), 0.5 + (0.1j if cplx else 0j), dtype=torch.complex128, device="cuda"),
                   torch.arange(n, dtype=torch.int32, device="cuda"), 1)
    c = [ctypes.c_int() for _ in range(3)]
    assert lib.kpm_ell_step_config(op.handle, _capi.KPM_C64, R, *map(ctypes.byref, c), None) == 0
    return tuple(x.value for x in c)


@pytest.mark.parametrize("upwards", [True, False])
def test_forms_at_the_limits(cuda_lib, upwards):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for cplx, R, n, kind, U in LIMITS if upwards else LIMITS[::-1]:
        got = _config(cuda_lib, n, R, cplx)
        assert got[:2] == (kind, U), (cplx, R, n)
        if not cplx and R == 1 and U == 1:
            assert got[2] == min(6 * sms, -(-n // 512) * 512 // 256)
        if not cplx and R == 8 and n >= 200000:
            assert got[2] == min(2 * sms, -(-n // 512) * 512 // 128)


@pytest.mark.parametrize("nx,ny,cplx,R", [(700, 520, False, 1), (900, 770, False, 1), (620, 500, True, 1), (500, 420, False, 8),
                                          (420, 400, True, 2)])
def test_moments_beyond(cuda_lib, nx, ny, cplx, R):
    import torch

    from minijclsquant_gb300 import device, lattice

    g = lattice.honeycomb_device(nx, ny, W=1.0, seed=1)
    n, L, data = g.n, g.len_row, g.data_kpm
    if cplx:  # a gauge: complex values, the same spectrum
        th = torch.from_numpy(np.random.default_rng(2).uniform(0, 6.28, n)).cuda()
        ph = torch.polar(torch.ones((n, L), dtype=torch.float64, device="cuda"), th[:, None] - th[g.indices.view(n, L).long()])
        data = (data.view(n, L) * ph).reshape(-1).contiguous()
    th = torch.from_numpy(np.random.default_rng(3).uniform(0, 6.28, (R, n))).cuda()
    v = torch.polar(torch.ones_like(th), th)
    mus = []
    for _ in range(2):
        op = device.DeviceELL(data, g.indices, L)
        mus.append(device.cheb_moments(op, 24, v, dtype="c64"))
        assert cuda_lib.kpm_ell_check(op.handle, None) == 0
    assert torch.equal(mus[0], mus[1])
    assert torch.max((mus[0] - device.cheb_moments(op, 24, v)).abs()).item() <= 2e-6 * n


def test_rows_too_wide_for_the_form_are_timed_once(cuda_lib):
    """Where the form by size does not fit the rows, the choice is timed and shared by later handles."""
    import torch

    from minijclsquant_gb300 import _capi
    from minijclsquant_gb300.device import DeviceELL

    n, L, R = 70001, 9, 2  # the staged kernel holds no two rows of nine complex slots
    i = torch.arange(n, device="cuda")
    idx = torch.stack([(i + 7 * s) % n for s in range(L)], dim=1).to(torch.int32).reshape(-1).contiguous()
    data = torch.full((n * L,), 0.05 + 0.01j, dtype=torch.complex128, device="cuda")
    seen = []
    for _ in range(3):
        op = DeviceELL(data, idx, L)
        c, us = [ctypes.c_int() for _ in range(3)], ctypes.c_float()
        assert cuda_lib.kpm_ell_step_config(op.handle, _capi.KPM_C64, R, *map(ctypes.byref, c), ctypes.byref(us)) == 0
        seen.append((*(x.value for x in c), us.value))
    assert seen[0] == seen[1] == seen[2] and seen[0][-1] > 0
