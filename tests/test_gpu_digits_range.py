"""The table contractions keep the error bound of FP64 products where large elements of one operand meet
small ones of the other, at the ends of the exponent range, and where no product is left.

A dot product of K terms in FP64 is within K 2^-53 T of the exact one, T = sum |a b|.  An output left to
the digits has T >= S / 4, S the sum over blocks of 512 of the operands' largest magnitudes (their
powers of two); a digit product errs by at most 2^-55 of a block's S, and joining a block's sums by
2^-54 of it and one rounding.  Both kinds of output are within (K + 4 blocks) 2^-53 T, but for 2^-9 of it
that the rounding of T takes, and K roundings of the smallest numbers."""
import numpy as np
import pytest

from test_gpu_digits import _gram, _handle, _mix

pytestmark = pytest.mark.gpu


def _bound(a, b):
    """(exact a b^T, its allowed error) of real operands [rows][K] in extended precision."""
    a, b = a.astype(np.longdouble), b.astype(np.longdouble)
    K = a.shape[1]
    per = np.longdouble(2) ** -53 * (K + 4 * ((K + 511) // 512)) * (1 + np.longdouble(2) ** -9)
    return a @ b.T, per * (np.abs(a) @ np.abs(b).T) + K * np.longdouble(2) ** -1074


def _reals(T):
    return np.ascontiguousarray(T).view(np.float64)


def _swapped(T):
    r = _reals(T).copy()
    r[:, 0::2], r[:, 1::2] = -_reals(T)[:, 1::2], _reals(T)[:, 0::2]
    return r


def _operands(kind, M, n, seed):
    rng = np.random.default_rng(seed)
    U, W = (rng.standard_normal((M, n)) + 1j * rng.standard_normal((M, n)) for _ in range(2))
    k = np.arange(n)
    if kind == "peaks":  # U is large where W is small, in every block
        U *= np.where(k % 7 == 0, 1.0, 1e-9)
        W *= np.where(k % 7 == 0, 1e-9, 1.0)
    elif kind == "decay":  # every row over its own number of decades, against each other
        U *= np.exp(-np.outer(rng.uniform(0, 60, M), k / n))
        W *= np.exp(-np.outer(rng.uniform(0, 60, M), 1 - k / n))
    elif kind == "lone":  # one product of ordinary size beside elements that meet zeros
        U[:, 1:] *= (k[1:] % 2)
        W[:, 1:] *= (1 - k[1:] % 2) * 1e12
    elif kind == "scales":  # rows from 2^-1000 to 2^1000
        s = np.ldexp(1.0, np.linspace(-1000, 1000, M).astype(int))
        U *= s[:, None]
        W *= s[::-1][:, None]
    elif kind == "real":  # imaginary parts zero: outputs without any product
        U, W = U.real + 0j, W.real + 0j
    return U, W


@pytest.mark.parametrize("kind", ["random", "peaks", "decay", "lone", "scales", "real"])
@pytest.mark.parametrize("M,n", [(3, 5), (40, 700), (131, 300)])
def test_gram_keeps_the_fp64_bound(cuda_lib, kind, M, n):
    h = _handle(n)
    U, W = _operands(kind, M, n, M + n)
    mu = _gram(cuda_lib, h, U, W).cpu().numpy()
    with np.errstate(over="ignore", invalid="ignore"):
        for rows, got in ((_reals(U), mu.real), (_swapped(U), mu.imag)):
            want, allowed = _bound(rows, _reals(W))
            held = np.abs(want) < 2.0 ** 1000  # beyond, a product of rows of 2^1000 overflows
            assert np.all(np.abs(got - want)[held] <= allowed[held])
    if kind == "real":
        assert np.all(mu.imag == 0)
    assert np.array_equal(mu, _gram(cuda_lib, h, U, W).cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("kind", ["random", "peaks", "decay", "lone", "scales"])
@pytest.mark.parametrize("M,n", [(3, 20), (24, 100), (257, 33), (600, 40)])
def test_mix_keeps_the_fp64_bound(cuda_lib, kind, M, n):
    h = _handle(n)
    A, B = _operands(kind, max(M, 2 * n), M, 3 * M + n)  # rows of C and columns of T over M orders
    C = np.ascontiguousarray(A.real[:M])
    T = np.ascontiguousarray((B.real[:n] + 1j * B.imag[n:2 * n]).T)
    Q = _mix(cuda_lib, h, C, T)
    with np.errstate(over="ignore", invalid="ignore"):
        for part in ("real", "imag"):
            want, allowed = _bound(C, np.ascontiguousarray(getattr(T, part).T))
            held = np.abs(want) < 2.0 ** 1000
            assert np.all(np.abs(getattr(Q, part) - want)[held] <= allowed[held])


def test_mix_of_a_peaked_matrix_is_no_worse_than_fp64(cuda_lib):
    """Rows of C peaked as those of a conductivity gradient are, against the FP64 library product."""
    import torch

    M, n = 64, 900
    h = _handle(n)
    rng = np.random.default_rng(2)
    m = np.arange(M)
    C = rng.standard_normal((M, M)) * np.exp(-np.abs(m[:, None] - m[None, :]) / 3.0)
    T = rng.standard_normal((M, n)) + 1j * rng.standard_normal((M, n))
    want = C.astype(np.longdouble) @ T.real.astype(np.longdouble)
    lib64 = (torch.from_numpy(C).cuda() @ torch.from_numpy(np.ascontiguousarray(T.real)).cuda()).cpu().numpy()
    rms = lambda x: float(np.sqrt(np.mean((x - want) ** 2)))  # noqa: E731
    assert rms(_mix(cuda_lib, h, C, T).real) <= rms(lib64)
