"""Table contractions of more orders than one block of them takes (rows of a gram, of a mix, columns of a
mix), on both sides of a block's edge, against FP64 library products: both are within K 2^-53 sum |a b| of
the exact value and half a unit more per block of 512."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,n", [(4096, 40), (4097, 9), (9001, 300), (16400, 36)])
def test_many_orders(cuda_lib, M, n):
    import torch

    from minijclsquant_gb300.device import DeviceELL

    h = DeviceELL(np.full(n, 0.5 + 0j), np.arange(n, dtype=np.int32), 1)
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    U, W = (torch.randn((M, n), dtype=torch.complex128, device="cuda", generator=g) for _ in range(2))
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert cuda_lib.kpm_table_work_bytes(h.handle, M) < 3e9
    mu = torch.full((M, M), float("nan"), dtype=torch.complex128, device="cuda")
    assert cuda_lib.kpm_table_gram(h.handle, M, U.data_ptr(), W.data_ptr(), 0, mu.data_ptr(), s) == 0
    per = lambda K: 2.0 ** -53 * 2 * (K + 4 * ((K + 511) // 512)) * 1.01  # noqa: E731
    u, w = torch.view_as_real(U).reshape(M, -1), torch.view_as_real(W).reshape(M, -1)
    swapped = torch.view_as_real(U * 1j).reshape(M, -1)
    for rows, got in ((u, mu.real), (swapped, mu.imag)):
        assert torch.all((got - rows @ w.T).abs() <= per(2 * n) * (rows.abs() @ w.abs().T))
    del mu
    C = torch.randn((M, M), dtype=torch.float64, device="cuda", generator=g)
    Q = torch.full_like(U, float("nan"))
    assert cuda_lib.kpm_table_mix(h.handle, M, C.data_ptr(), U.data_ptr(), Q.data_ptr(), s) == 0
    q = torch.view_as_real(Q).reshape(M, -1)
    assert torch.all((q - C @ u).abs() <= per(M) * (C.abs() @ u.abs()))
    assert cuda_lib.kpm_ell_check(h.handle, None) == 0
