"""Vector tables as one cooperative launch against the step launches, which a captured call takes.

Both add the same products in the same order, so the results are equal bit for bit; with an all-imaginary
second operator the cooperative kernel leaves out products with zero, which changes no value but may
change the sign of a zero (equal under ==).  Infinities and NaN stay where they were."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _op(lib, val, idx, L):
    h = ctypes.c_void_p()
    n = idx.size // L
    assert lib.kpm_ell_create(ctypes.byref(h), n, L, val.ctypes.data, idx.ctypes.data, 0, None) == 0
    return h


def _values(rng, size, kind):
    a, b = rng.uniform(-0.4, 0.4, size), rng.uniform(-0.4, 0.4, size)
    return {"real": a + 0j, "imag": 1j * b, "complex": a + 1j * b}[kind]


def _same(a, b):
    a, b = a.cpu().numpy().view(np.float64), b.cpu().numpy().view(np.float64)
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("n,Lh,Ls", [(1, 1, 1), (7, 3, 5), (64, 4, 4), (65, 5, 1), (9731, 3, 5), (131073, 4, 4),
                                     (152 * 1536, 1, 1), (152 * 1536 + 1, 2, 1)])
@pytest.mark.parametrize("kh,ks", [("real", "imag"), ("complex", "real"), ("complex", "complex"), ("real", None)])
@pytest.mark.parametrize("M", [3, 4, 9])
def test_resident_tables_equal_steps(cuda_lib, n, Lh, Ls, kh, ks, M):
    import torch

    rng = np.random.default_rng(n + Lh)
    idx_h = rng.integers(0, n, n * Lh).astype(np.int32) if n < 5000 else (
        (np.arange(n)[:, None] + rng.integers(-700, 700, (1, Lh))) % n).astype(np.int32).ravel()
    idx_s = rng.integers(0, n, n * Ls).astype(np.int32)
    h = _op(cuda_lib, _values(rng, n * Lh, kh), idx_h, Lh)
    s = _op(cuda_lib, _values(rng, n * Ls, ks), idx_s, Ls) if ks else None
    z = torch.from_numpy(rng.normal(size=(M, n)) + 1j * rng.normal(size=(M, n))).cuda()
    z_inf = z.clone()
    z_inf[:, n // 2] = complex(np.inf, 0.0)

    def run(x):
        stream = torch.cuda.current_stream().cuda_stream
        tab, stab, lam = (torch.empty_like(x) for _ in range(3))
        assert cuda_lib.kpm_cheb_table(h, s, M, x.data_ptr(), tab.data_ptr(), stab.data_ptr() if s else None,
                                       stream) == 0
        assert cuda_lib.kpm_cheb_clenshaw_table(h, s, M, x.data_ptr(), lam.data_ptr(), stream) == 0
        return [tab, lam] + ([stab] if s else [])

    try:
        for x in (z, z_inf):
            got = run(x)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                want = run(x)
            g.replay()
            torch.cuda.synchronize()
            assert all(_same(a, b) for a, b in zip(got, want))
            # calls under way on two streams of one handle
            streams = [torch.cuda.Stream() for _ in range(2)]
            both = []
            for st in streams:
                with torch.cuda.stream(st):
                    both.append(run(x))
            torch.cuda.synchronize()
            assert all(_same(a, b) for res in both for a, b in zip(res, want))
        assert cuda_lib.kpm_ell_check(h, None) == 0
    finally:
        cuda_lib.kpm_ell_destroy(h)
        if s:
            cuda_lib.kpm_ell_destroy(s)
