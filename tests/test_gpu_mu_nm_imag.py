"""The fused right step of kpm_mu_nm with an all-imaginary velocity against the general product.

One entry of V given a real part of 1e-30 sends every row through the general product and changes no
rounded result: the products it adds to are of order 1e-3 and rounded to 24 bits.  The two moment
matrices are then equal bit for bit; infinite inputs end as NaN in the same places."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,peierls", [(3, 2, 0.0), (40, 30, 0.0), (61, 47, 0.0), (40, 30, 1.3)])
@pytest.mark.parametrize("R", [1, 2, 4, 5])
def test_imaginary_velocity_equals_general(cuda_lib, nx, ny, peierls, R):
    import torch

    from minijclsquant_gb300 import _capi, device, lattice
    from minijclsquant_gb300.modifiers import modifier_bounds, modifier_velocity
    from minijclsquant_gb300.observables import random_vector_generator

    H = lattice.honeycomb(nx, ny, t=-2.7, W=1.0, seed=8)
    Hk = H.modifier(modifier_bounds)
    Vi = H.modifier(modifier_velocity, "x").data / H.bounds[1]
    data = Hk.data * np.exp(1e-3j * peierls * np.arange(Hk.data.size))  # complex H values: the other kernel
    Vi = 1j * Vi.imag
    Vm = Vi.copy()
    Vm[np.argmax(np.abs(Vm))] += 1e-30
    Nm, n = 33, H.shape[0]
    vs = np.stack([random_vector_generator(n, 70 + r) for r in range(R)])
    for x in (vs, np.where(np.arange(n) == n // 2, np.inf, vs)):
        out = []
        for V in (Vi, Vm):
            hop = device.DeviceELL(data, Hk.indices, Hk.len_row)
            vop = device.DeviceELL(V, Hk.indices, Hk.len_row)
            mu = torch.empty((Nm, Nm), dtype=torch.complex128, device="cuda")
            tx = torch.from_numpy(x).cuda()
            st = cuda_lib.kpm_mu_nm(hop.handle, vop.handle, R, Nm, tx.data_ptr(), mu.data_ptr(), None)
            assert st == 0, _capi.lib().kpm_strerror(st)
            assert cuda_lib.kpm_ell_check(hop.handle, None) == 0
            out.append(mu.cpu().numpy().view(np.float64))
        assert np.array_equal(out[0], out[1], equal_nan=True)
