"""kpm_table_gram / kpm_table_mix (exact digit products on the tensor cores) against extended
precision, at the edges of their tiles (128 x 64 outputs, 512-element blocks, 32-element stages).

The bound follows from the digits: an element is off by at most 2^-55 of its block's largest
magnitude, and the digit pairs left out of a product are worth at most 2^-51 of the two block
maxima, so a sum of K products is within K 2^-50 max|a| max|b| (block sums are exact; adding
them rounds once per 512 products).  On random tables the error is also compared with that of
the FP64 library product, which it may not exceed.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _handle(n):
    from minijclsquant_gb300.device import DeviceELL

    return DeviceELL(np.full(n, 0.5 + 0j), np.arange(n, dtype=np.int32), 1)


def _tables(M, n, seed, count=2):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal((M, n)) + 1j * rng.standard_normal((M, n)) for _ in range(count)]


def _gram(lib, h, U, W, accumulate=0, mu=None):
    import torch

    u, w = torch.from_numpy(U).cuda(), torch.from_numpy(W).cuda()
    mu = torch.empty((U.shape[0],) * 2, dtype=torch.complex128, device="cuda") if mu is None else mu
    st = lib.kpm_table_gram(h.handle, U.shape[0], u.data_ptr(), w.data_ptr(), accumulate, mu.data_ptr(),
                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    assert lib.kpm_ell_check(h.handle, ctypes.c_void_p(0)) == 0
    return mu


def _mix(lib, h, C, T):
    import torch

    c, t = torch.from_numpy(C).cuda(), torch.from_numpy(T).cuda()
    q = torch.full_like(t, float("nan"))
    st = lib.kpm_table_mix(h.handle, T.shape[0], c.data_ptr(), t.data_ptr(), q.data_ptr(),
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    assert lib.kpm_ell_check(h.handle, ctypes.c_void_p(0)) == 0
    return q.cpu().numpy()


def _ext(a, b):
    """Real a b^T in extended precision for the rows of a and b."""
    return a.astype(np.longdouble) @ b.astype(np.longdouble).T


def _gram_ext(U, W):
    re = _ext(U.real, W.real) + _ext(U.imag, W.imag)
    im = _ext(U.real, W.imag) - _ext(U.imag, W.real)
    return re, im


def _amax(T):
    return np.max(np.maximum(np.abs(T.real), np.abs(T.imag)), axis=1)


@pytest.mark.parametrize("M,n", [(1, 1), (2, 15), (3, 16), (24, 17), (63, 255), (64, 256), (65, 257), (128, 300),
                                 (129, 33), (256, 100), (7, 40000)])
def test_gram_and_mix_within_the_digit_bound(cuda_lib, M, n):
    import torch

    h = _handle(n)
    U, W = _tables(M, n, 7 * M + n)
    U[M // 2] *= 1e-30  # every row has its own scale
    W[0] *= 1e25
    mu = _gram(cuda_lib, h, U, W).cpu().numpy()
    rows = np.arange(M) if M <= 65 and n < 1000 else np.unique(np.linspace(0, M - 1, 9).astype(int))
    re, im = _gram_ext(U[rows], W)
    bound = 2 * n * 2.0 ** -50 * np.outer(_amax(U[rows]), _amax(W))
    assert np.all(np.abs(mu[rows].real - re) <= bound) and np.all(np.abs(mu[rows].imag - im) <= bound)
    twice = _gram(cuda_lib, h, U, W, 1, torch.from_numpy(mu).cuda()).cpu().numpy()
    assert np.array_equal(twice, 2 * mu)  # accumulation; a second run is bit-identical
    C = np.random.default_rng(M).standard_normal((M, M)) * np.logspace(0, -6, M)[:, None]
    Q = _mix(cuda_lib, h, C, U)
    cols = np.arange(n) if n <= 300 else np.unique(np.linspace(0, n - 1, 200).astype(int))
    for part in ("real", "imag"):
        t = np.ascontiguousarray(getattr(U, part)[:, cols])
        bound = M * 2.0 ** -50 * np.outer(np.max(np.abs(C), axis=1), np.max(np.abs(t), axis=0))
        assert np.all(np.abs(getattr(Q, part)[:, cols] - _ext(C, t.T)) <= bound)


def test_error_is_no_larger_than_the_fp64_product(cuda_lib):
    import torch

    M, n = 96, 3000
    h = _handle(n)
    U, W = _tables(M, n, 5)
    re, im = _gram_ext(U[:12], W)
    lib64 = (torch.from_numpy(U).cuda().conj() @ torch.from_numpy(W).cuda().T).cpu().numpy()
    mu = _gram(cuda_lib, h, U, W).cpu().numpy()
    rms = lambda x: float(np.sqrt(np.mean((x[:12].real - re) ** 2 + (x[:12].imag - im) ** 2)))  # noqa: E731
    assert rms(mu) <= rms(lib64)
    C = np.random.default_rng(3).standard_normal((M, M))
    q64 = (torch.from_numpy(C).cuda() @ torch.from_numpy(np.ascontiguousarray(U.real)).cuda()).cpu().numpy()
    q = _mix(cuda_lib, h, C, U).real
    ref = _ext(C[:12], np.ascontiguousarray(U.real.T))
    rms = lambda x: float(np.sqrt(np.mean((x[:12] - ref) ** 2)))  # noqa: E731
    assert rms(q) <= rms(q64)


def test_zero_and_non_finite_rows(cuda_lib):
    M, n = 20, 700
    h = _handle(n)
    U, W = _tables(M, n, 11)
    U[3] = 0
    W[5, 650] = np.nan
    W[6, 2] = np.inf
    mu = _gram(cuda_lib, h, U, W).cpu().numpy()
    assert np.all(mu[3, :5] == 0)
    assert np.all(np.isnan(mu[:, 5])) and np.all(np.isnan(mu[:, 6]))
    ok = [m for m in range(M) if m not in (5, 6)]
    assert np.all(np.isfinite(mu[:, ok]))
    Q = _mix(cuda_lib, h, np.ones((M, M)), W)
    assert np.all(np.isnan(Q.real[:, [2, 650]])) and np.all(np.isfinite(np.delete(Q, [2, 650], axis=1)))
