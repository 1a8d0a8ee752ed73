"""Two moment sets by the producer-warp step against the grid-stride step, complex128.

Both form the same T_m; only the order of the FP64 sums over the n sites differs.  With a Hermitian H of
norm <= 1, sum_i |l_i T_m,i| <= |l| |T_m| <= |l| |v|, so two orders of the 2 n products of a part agree to
2 (2 n + 8) u |l| |v| with u = 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (16, 8), (37, 29), (200, 170)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("R", [1, 2, 4, 8, 3])
def test_two_sets_equal_grid_stride(cuda_lib, monkeypatch, nx, ny, cplx, R):
    import torch

    from minijclsquant_gb300 import device, lattice
    from minijclsquant_gb300.modifiers import modifier_bounds
    from minijclsquant_gb300.observables import random_vector_generator

    H = lattice.honeycomb(nx, ny, t=-2.7, W=0.7, seed=5)
    Hk = H.modifier(modifier_bounds)
    n, L = H.shape[0], Hk.len_row
    data = Hk.data
    if cplx:  # a gauge: the same spectrum with complex values
        th = np.random.default_rng(1).uniform(0, 6.28, n)
        data = data * np.exp(1j * (np.repeat(th, L) - th[Hk.indices]))
    vr, vl = (np.stack([random_vector_generator(n, s + r) for r in range(R)]) for s in (70, 90))
    M = 70  # more than one chunk of partials
    res = {}
    for kernel in ("simple", "ws1"):
        monkeypatch.setenv("KPM_STEP_KERNEL", kernel)
        op = device.DeviceELL(data, Hk.indices, L)
        mu, rr = (torch.empty((R, M), dtype=torch.complex128, device="cuda") for _ in range(2))
        tr, tl = torch.from_numpy(vr).cuda(), torch.from_numpy(vl).cuda()
        assert cuda_lib.kpm_cheb_moments(op.handle, 0, R, M, tr.data_ptr(), tl.data_ptr(), mu.data_ptr(),
                                         rr.data_ptr(), None) == 0
        assert cuda_lib.kpm_ell_check(op.handle, None) == 0
        res[kernel] = [mu.cpu().numpy(), rr.cpu().numpy()]
    for k, left in enumerate((vl, vr)):
        tol = 2 * (2 * n + 8) * 2.0**-53 * np.linalg.norm(left, axis=1) * np.linalg.norm(vr, axis=1)
        assert np.all(np.abs(res["ws1"][k] - res["simple"][k]) <= 2 * tol[:, None])
