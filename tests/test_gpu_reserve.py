"""After kpm_ell_reserve a moment call allocates nothing, so it can be recorded into a graph straight away: for
operators whose recursion is one launch and for larger ones, for every group that the vectors are cut into,
one moment set and two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("nx,ny,R,M", [(12, 10, 1, 2), (12, 10, 3, 8), (40, 36, 8, 40), (220, 200, 2, 9), (700, 430, 3, 12)])
def test_calls_after_reserve_allocate_nothing(cuda_lib, dtype, nx, ny, R, M):
    import torch

    from minijclsquant_gb300 import device, lattice

    g = lattice.honeycomb_device(nx, ny, W=1.0, seed=1)
    th = torch.from_numpy(np.random.default_rng(4).uniform(0, 6.28, (2, R, g.n))).cuda()
    v, vl = torch.polar(torch.ones_like(th), th)
    g.op.reserve(dtype, R, M)
    held = g.op.device_bytes()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        one = device.cheb_moments(g.op, M, v, dtype=dtype)
        two = device.cheb_moments(g.op, M, v, v_l=vl, dtype=dtype, both=True)
    graph.replay()
    torch.cuda.synchronize()
    assert g.op.device_bytes() == held
    assert torch.equal(one, device.cheb_moments(g.op, M, v, dtype=dtype))
    want = device.cheb_moments(g.op, M, v, v_l=vl, dtype=dtype, both=True)
    assert torch.equal(two[0], want[0]) and torch.equal(two[1], want[1])
    assert cuda_lib.kpm_ell_check(g.op.handle, None) == 0
