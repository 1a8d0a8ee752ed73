"""The real and imaginary per-slot sums (kpm_ell_slot_sum_part) against NumPy, at the slot counts where
the kernel's register tile changes and one row beyond a block.

Tolerance: K terms of two products each, summed in float64 in either order, differ from the exact sum
by at most (2 K + 2) u sum_k |c_k A_k B_k| (twice that between two such sums), u = 2^-53; the factor
sqrt 2 covers |re re| + |im im| <= 2 |A| |B| / sqrt 2."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,n", [(1, 1), (3, 257), (4, 256), (5, 300), (8, 513), (9, 64), (16, 255)])
@pytest.mark.parametrize("K,weighted", [(1, False), (6, True)])
def test_slot_sum_part(cuda_lib, L, n, K, weighted):
    import torch

    rng = np.random.default_rng(L * 100 + K)
    idx = rng.integers(0, n, n * L).astype(np.int32)
    val = rng.normal(size=n * L) + 0j
    lda = n + 2
    A, B = (rng.normal(size=(K, lda)) + 1j * rng.normal(size=(K, lda)) for _ in range(2))
    c = rng.uniform(0.5, 2.0, K) if weighted else np.ones(K)
    term = (c[:, None] * np.conj(A[:, :n]))[:, :, None] * B[:, idx.reshape(n, L)]
    bound = 2 * (2 * K + 2) * 2.0**-53 * np.sqrt(2.0) * np.abs(term).sum(0)
    base = rng.normal(size=(n, L))
    ta, tb, tc = (torch.from_numpy(x).cuda() for x in (A, B, c))
    h = ctypes.c_void_p()
    assert cuda_lib.kpm_ell_create(ctypes.byref(h), n, L, val.ctypes.data, idx.ctypes.data, 0, None) == 0
    try:
        for imag, ref in ((0, term.real.sum(0)), (1, term.imag.sum(0))):
            for acc in (0, 1):
                out = torch.from_numpy(base.copy()).cuda()
                assert cuda_lib.kpm_ell_slot_sum_part(h, K, tc.data_ptr() if weighted else None, ta.data_ptr(), lda,
                                                      tb.data_ptr(), lda, imag, acc, out.data_ptr(), None) == 0
                torch.cuda.synchronize()
                want = ref + acc * base
                tol = bound + acc * (2 * K + 2) * 2.0**-52 * np.abs(base)
                assert np.all(np.abs(out.cpu().numpy() - want) <= tol)
    finally:
        cuda_lib.kpm_ell_destroy(h)
