"""Recursions replayed as a graph at the sizes that the one-launch form leaves to it, against the same
steps launched one by one: bit-identical."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,nx,ny,R", [("c128", 600, 500, 1), ("c128", 380, 350, 3), ("c64", 220, 200, 1),
                                          ("c64", 260, 250, 5)])
def test_graph_equals_launches(cuda_lib, dtype, nx, ny, R):
    import torch

    from minijclsquant_gb300 import device, lattice

    g = lattice.honeycomb_device(nx, ny, W=1.0, seed=4)
    th = torch.from_numpy(np.random.default_rng(6).uniform(0, 6.28, (2, R, g.n))).cuda()
    v = torch.polar(torch.ones_like(th), th)
    got = [device.cheb_moments(g.op, 40, v[i].contiguous(), dtype=dtype).cpu().numpy() for i in range(2)]
    os.environ["KPM_NO_GRAPH"] = "1"
    try:
        want = [device.cheb_moments(g.op, 40, v[i].contiguous(), dtype=dtype).cpu().numpy() for i in range(2)]
    finally:
        del os.environ["KPM_NO_GRAPH"]
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
