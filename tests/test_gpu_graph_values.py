"""Recursions replayed as a graph after the operator's values change, at sizes that the one-launch form leaves
to the graph: the recorded kernels must read the new values (and the complex64 copy that is rebuilt), also
after a call that grew the buffers it was recorded with.  Bit for bit as the same steps launched one by one,
and as a new operator of the new values."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _direct(fn):
    os.environ["KPM_NO_GRAPH"] = "1"
    try:
        return fn()
    finally:
        del os.environ["KPM_NO_GRAPH"]


@pytest.mark.parametrize("dtype,nx,ny,R", [("c128", 560, 500, 1), ("c64", 210, 200, 1), ("c64", 180, 160, 3)])
def test_replay_after_new_values(cuda_lib, dtype, nx, ny, R):
    import ctypes

    import torch

    from minijclsquant_gb300 import _capi, device, lattice

    g = lattice.honeycomb_device(nx, ny, W=1.0, seed=4)
    th = torch.from_numpy(np.random.default_rng(6).uniform(0, 6.28, (8, g.n))).cuda()
    vs = torch.polar(torch.ones_like(th), th)
    v, M = vs[:R].contiguous(), 40
    run = lambda op: device.cheb_moments(op, M, v, dtype=dtype)  # noqa: E731
    first = run(g.op)
    c = [ctypes.c_int64(), ctypes.c_int64()]
    assert cuda_lib.kpm_ell_one_launch_counts(g.op.handle, *map(ctypes.byref, c)) == 0
    assert torch.equal(first, run(g.op)) and torch.equal(first, _direct(lambda: run(g.op)))
    for scale in (0.5, 0.25):
        data = (g.data_kpm * scale).contiguous()
        assert cuda_lib.kpm_ell_set_values(g.op.handle, data.data_ptr(), _capi.KPM_FLAG_DEVICE_PTRS, None) == 0
        torch.cuda.synchronize()
        got = run(g.op)
        assert not torch.equal(got, first)
        assert torch.equal(got, _direct(lambda: run(g.op)))
        assert torch.equal(got, run(device.DeviceELL(data, g.indices, g.len_row)))
        device.cheb_moments(g.op, 300, vs, dtype=dtype)  # larger buffers
        assert torch.equal(got, run(g.op))
    if R == 1:
        assert c[0].value == 0  # not the one-launch form
    assert cuda_lib.kpm_ell_check(g.op.handle, None) == 0
