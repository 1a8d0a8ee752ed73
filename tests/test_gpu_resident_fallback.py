"""A context with fewer SMs than the launch was shaped for refuses the one-launch forms (nothing runs), and
the step launches serve the call: the moments to the order of their sums (4 n 2^-53 ||v_l|| ||T_m v|| as in
test_gpu_resident; ||T_m v|| <= ||v|| here, 2^-40 of that for the recursion's rounding), the tables equal.
Sizes: a share of 256 CTAs (their limit) takes more than half an SM's shared memory."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fewer_sms(lib, op, call):
    """(call(), call() shaped for more SMs than there are, call())."""
    from minijclsquant_gb300 import _capi

    first = call()
    assert lib.kpm_ell_test_sm_count(None, 1) == _capi.KPM_ERR_INVALID_ARG
    assert lib.kpm_ell_test_sm_count(op.handle, 1000) == 0
    try:
        refused = call()
    finally:
        assert lib.kpm_ell_test_sm_count(op.handle, 0) == 0
    last = call()
    assert lib.kpm_ell_check(op.handle, None) == 0
    return first, refused, last


@pytest.mark.parametrize("nx,ny,R", [(400, 388, 1), (250, 250, 4)])
def test_moments(cuda_lib, nx, ny, R):
    import torch

    from minijclsquant_gb300 import device, lattice

    g = lattice.honeycomb_device(nx, ny, W=1.0, seed=5)
    th = torch.from_numpy(np.random.default_rng(1).uniform(0, 6.28, (R, g.n))).cuda()
    v = torch.polar(torch.ones_like(th), th)
    a, b, c = _fewer_sms(cuda_lib, g.op, lambda: device.cheb_moments(g.op, 24, v))
    assert torch.max((a - b).abs()).item() <= (4 * g.n * 2.0 ** -53 + 2.0 ** -40) * g.n
    assert torch.equal(a, c)


def test_tables(cuda_lib):
    import torch

    from minijclsquant_gb300 import device, lattice

    g = lattice.honeycomb_device(400, 290, W=1.0, seed=5)
    s_op = device.DeviceELL(g.data_kpm, g.indices, g.len_row)
    v = torch.randn((1, g.n), dtype=torch.complex128, device="cuda")
    M = 12

    def tables():
        t = [torch.empty((M, g.n), dtype=torch.complex128, device="cuda") for _ in range(3)]
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert cuda_lib.kpm_cheb_table(g.op.handle, s_op.handle, M, v.data_ptr(), t[0].data_ptr(), t[1].data_ptr(), s) == 0
        assert cuda_lib.kpm_cheb_clenshaw_table(g.op.handle, s_op.handle, M, t[1].data_ptr(), t[2].data_ptr(), s) == 0
        return t

    for t in zip(*_fewer_sms(cuda_lib, g.op, tables)):
        assert torch.equal(t[0], t[1]) and torch.equal(t[0], t[2])
