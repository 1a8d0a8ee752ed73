"""That the one-launch forms ran where they should and nowhere else, on both sides of their limits, and what
becomes of a wait between their CTAs that runs out (kpm_ell_test_withhold: the first CTA stops publishing,
every wait has a short limit; nothing hangs or faults)."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return min(256, torch.cuda.get_device_properties(0).multi_processor_count)


def _counts(lib, op):
    c = [ctypes.c_int64(), ctypes.c_int64()]
    assert lib.kpm_ell_one_launch_counts(op.handle, *map(ctypes.byref, c)) == 0
    return [x.value for x in c]


def _diag(n):
    import torch

    from minijclsquant_gb300.device import DeviceELL

    return DeviceELL(torch.full((n,), 0.5 + 0j, dtype=torch.complex128, device="cuda"),
                     torch.arange(n, dtype=torch.int32, device="cuda"), 1)


@pytest.mark.parametrize("dtype,R,size,fits", [("c128", 1, lambda s: 3500 * s, True), ("c128", 1, lambda s: 3500 * s + 1, False),
                                               ("c128", 4, lambda s: 875 * s, True), ("c128", 4, lambda s: 875 * s + 1, False),
                                               ("c64", 1, lambda s: 80000, True), ("c64", 1, lambda s: 80001, False),
                                               ("c64", 8, lambda s: 10000, True), ("c64", 8, lambda s: 10001, False)])
def test_moments_at_the_limits(cuda_lib, dtype, R, size, fits):
    import torch

    from minijclsquant_gb300 import device

    n = size(_sms())
    op = _diag(n)
    v = torch.ones((R, n), dtype=torch.complex128, device="cuda")
    mu = device.cheb_moments(op, 5, v, dtype=dtype)
    assert _counts(cuda_lib, op) == [1 if fits else 0, 0]
    want = n * torch.cos(torch.arange(5, device="cuda", dtype=torch.float64) * np.pi / 3)  # T_m(1 / 2)
    assert torch.max((mu - want[None, :]).abs()).item() <= n * (1e-12 if dtype == "c128" else 1e-6)


@pytest.mark.parametrize("M,size,fits", [(4, lambda s: 1536 * s, True), (3, lambda s: 1000, False),
                                         (4, lambda s: 1536 * s + 1, False)])
def test_tables_at_the_limits(cuda_lib, M, size, fits):
    import torch

    n = size(_sms())
    op = _diag(n)
    z = torch.ones((M, n), dtype=torch.complex128, device="cuda")
    tab, lam = torch.empty_like(z), torch.empty_like(z)
    assert cuda_lib.kpm_cheb_table(op.handle, None, M, z.data_ptr(), tab.data_ptr(), None, None) == 0
    assert cuda_lib.kpm_cheb_clenshaw_table(op.handle, None, M, z.data_ptr(), lam.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert _counts(cuda_lib, op) == [0, 2 if fits else 0]
    want = torch.cos(torch.arange(M, device="cuda", dtype=torch.float64) * np.pi / 3)
    assert torch.max((tab - want[:, None]).abs()).item() <= 1e-14
    assert abs(lam[0, n - 1].item() - want.sum().item()) <= 1e-13


@pytest.mark.parametrize("order", [0, 1, 6])
@pytest.mark.parametrize("dtype,R", [("c128", 1), ("c128", 4), ("c64", 2)])
def test_moments_whose_wait_runs_out(cuda_lib, dtype, R, order):
    import torch

    from minijclsquant_gb300 import _capi, device, lattice

    g = lattice.honeycomb_device(40, 35, W=1.0, seed=3)
    op = g.op
    v = torch.ones((R, g.n), dtype=torch.complex128, device="cuda")
    want = device.cheb_moments(op, 20, v, dtype=dtype)
    assert cuda_lib.kpm_ell_test_withhold(op.handle, 10, order) == _capi.KPM_ERR_INVALID_ARG
    assert cuda_lib.kpm_ell_test_withhold(op.handle, 20_000_000, order) == 0
    try:
        t0 = time.perf_counter()
        mu = device.cheb_moments(op, 20, v, dtype=dtype)
        assert cuda_lib.kpm_ell_check(op.handle, None) == _capi.KPM_ERR_TIMEOUT
        assert time.perf_counter() - t0 < 5.0
    finally:
        assert cuda_lib.kpm_ell_test_withhold(op.handle, 0, -1) == 0
    assert torch.all(torch.isnan(mu[:, order + 2:].real))
    assert cuda_lib.kpm_ell_check(op.handle, None) == 0
    assert torch.equal(device.cheb_moments(op, 20, v, dtype=dtype), want)
    assert _counts(cuda_lib, op)[0] == 3


@pytest.mark.parametrize("order", [0, 3])
def test_tables_whose_wait_runs_out(cuda_lib, order):
    import torch

    from minijclsquant_gb300 import _capi, device, lattice

    g = lattice.honeycomb_device(40, 35, W=1.0, seed=3)
    s_op = device.DeviceELL(1j * g.data_kpm, g.indices, g.len_row)
    M = 9
    z = torch.ones((M, g.n), dtype=torch.complex128, device="cuda")

    def tables():
        t = [torch.empty_like(z) for _ in range(3)]
        assert cuda_lib.kpm_cheb_table(g.op.handle, s_op.handle, M, z.data_ptr(), t[0].data_ptr(), t[1].data_ptr(), None) == 0
        first = cuda_lib.kpm_ell_check(g.op.handle, None)
        assert cuda_lib.kpm_cheb_clenshaw_table(g.op.handle, s_op.handle, M, z.data_ptr(), t[2].data_ptr(), None) == 0
        return t, (first, cuda_lib.kpm_ell_check(g.op.handle, None))

    torch.cuda.synchronize()
    want, status = tables()
    assert status == (0, 0)
    assert cuda_lib.kpm_ell_test_withhold(g.op.handle, 20_000_000, order) == 0
    try:
        t0 = time.perf_counter()
        _, status = tables()
        assert status == (_capi.KPM_ERR_TIMEOUT, _capi.KPM_ERR_TIMEOUT)
        assert time.perf_counter() - t0 < 5.0
    finally:
        assert cuda_lib.kpm_ell_test_withhold(g.op.handle, 0, -1) == 0
    got, status = tables()
    assert status == (0, 0) and all(torch.equal(a, b) for a, b in zip(got, want))
