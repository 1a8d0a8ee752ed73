"""Whole recursions as one cooperative launch (kpm_resident.cu) against the step launches
(KPM_STEP_KERNEL=simple), at the edges of the row split: one row, fewer rows than CTAs, a ragged
last CTA, wide rows, every vector group, operators whose CTAs all depend on each other, one-way
patterns (a CTA that is read by others but reads none of them), both value types, one and two
moment sets, and sizes on both sides of the fit.

T_m is computed by the same operations in the same order, so moments differ only by the order
of their sums: at most 4 n 2^-53 ||v_l|| ||T_m v|| in complex128, and 24 * 2^-24 of that product of
norms in complex64, whose products are summed in float over 8 rows.  The patterns are not
symmetric, so ||T_m v|| may grow with m; it is taken from a plain FP64 recursion.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pattern(kind, n, seed):
    """(data, indices, L) with every absolute row sum below one."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    if kind == "ring":  # neighbours at distances 1 and 37
        cols = np.stack([i, (i + 1) % n, (i - 1) % n, (i + 37) % n, (i - 37) % n], axis=1)
    elif kind == "random":  # every CTA needs every other
        cols = rng.integers(0, n, (n, 6))
    elif kind == "oneway":  # row i reads rows ahead of it only
        cols = np.stack([i, np.minimum(i + 1, n - 1), np.minimum(i + n // 2, n - 1)], axis=1)
    else:  # wide
        cols = rng.integers(0, n, (n, 19))
    L = cols.shape[1]
    vals = rng.uniform(-1, 1, (n, L)) / L
    return vals, cols.astype(np.int32), L


def _both(fn):
    out = fn()
    os.environ["KPM_STEP_KERNEL"] = "simple"
    try:
        return out, fn()
    finally:
        del os.environ["KPM_STEP_KERNEL"]


def _norms(data, cols, v, M):
    """||T_m v_r||, [R, M], by a plain recursion in torch."""
    import torch

    d = torch.from_numpy(np.ascontiguousarray(data)).to(torch.complex128).cuda()
    c = torch.from_numpy(cols.astype(np.int64)).cuda()
    mul = lambda x: sum(d[:, s] * x[:, c[:, s]] for s in range(d.shape[1]))  # noqa: E731
    t0, t1, out = v, mul(v), [v.norm(dim=1)]
    for _ in range(M - 1):
        out.append(t1.norm(dim=1))
        t0, t1 = t1, 2 * mul(t1) - t0
    return torch.stack(out, dim=1)


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("kind,n,R", [("ring", 1, 1), ("ring", 100, 1), ("ring", 151, 8), ("ring", 9729, 1),
                                      ("ring", 30011, 4), ("random", 5000, 2), ("random", 20001, 3),
                                      ("oneway", 20000, 1), ("oneway", 4097, 8), ("wide", 3000, 4),
                                      ("ring", 65537, 8), ("ring", 140001, 2), ("ring", 200003, 4)])
@pytest.mark.parametrize("cplx", [False, True])
def test_resident_equals_step_launches(cuda_lib, kind, n, R, dtype, cplx):
    import torch

    from minijclsquant_gb300 import device

    vals, cols, L = _pattern(kind, n, n + R)
    rng = np.random.default_rng(n)
    data = vals * np.exp(1j * rng.uniform(0, 6, vals.shape)) if cplx else vals + 0j
    op = device.DeviceELL(data.reshape(-1), cols.reshape(-1), L)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    v = torch.randn((R, n), dtype=torch.complex128, device="cuda", generator=g)
    vl = torch.randn((R, n), dtype=torch.complex128, device="cuda", generator=g)
    tol = (4 * n * 2.0 ** -53) if dtype == "c128" else 24 * 2.0 ** -24
    norms = _norms(data, cols, v, 34)
    for M in (2, 3, 34):
        for kw in ({}, {"v_l": vl}, {"v_l": vl, "both": True}):
            a, b = _both(lambda: device.cheb_moments(op, M, v, dtype=dtype, **kw))
            again = device.cheb_moments(op, M, v, dtype=dtype, **kw)
            a, b, again = (x if isinstance(x, tuple) else (x,) for x in (a, b, again))
            lefts = (kw.get("v_l", v), v)
            for x, y, z, left in zip(a, b, again, lefts):
                assert torch.equal(x, z)
                scale = left.norm(dim=1)[:, None] * norms[:, :M]
                assert torch.all((x - y).abs() <= tol * scale), (M, kw.keys())
    torch.cuda.synchronize()
