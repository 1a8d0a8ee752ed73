"""The float-float adjoint (KPM_C128F) against the FP64 one over row widths around its groups of
four slots, every vector count, and row counts around its tiles.

Both run the same recursion; float-float sums round at 2^-48, so after M orders of L slots and R
vectors the gradients agree to 16 L M 2^-48 of the largest entry.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operator(n, L, seed):
    """Real symmetric ELL: circulant bonds of random sign patterns, row sums below one."""
    rng = np.random.default_rng(seed)
    cols, vals = [np.arange(n)], [rng.uniform(-1, 1, n)]
    while len(cols) < L:
        k = len(cols) // 2 + 1
        w = rng.uniform(-1, 1, n)  # bond i -> i + k
        cols.append((np.arange(n) + k) % n)
        vals.append(w)
        if len(cols) < L:
            cols.append((np.arange(n) - k) % n)
            vals.append(np.roll(w, k))
    return (np.stack(vals, 1) / (2 * L)).astype(np.complex128), np.stack(cols, 1).astype(np.int32)


@pytest.mark.parametrize("L", [1, 3, 4, 5, 9])
@pytest.mark.parametrize("n,R", [(97, 1), (512, 2), (700, 4), (1300, 8)])
def test_float_float_adjoint_matches_fp64(cuda_lib, n, L, R):
    import torch

    from minijclsquant_gb300 import _capi, device

    data, cols = _operator(n, L, n + L)
    op = device.DeviceELL(data.reshape(-1), cols.reshape(-1), L)
    M, ckpt = 41, 7
    g = torch.Generator(device="cuda")
    g.manual_seed(L)
    v = torch.randn((R, n), dtype=torch.complex128, device="cuda", generator=g)
    c = torch.randn(M, dtype=torch.float64, device="cuda", generator=g)
    mu = torch.empty((R, M), dtype=torch.complex128, device="cuda")
    out = []
    for dtype in (_capi.KPM_C128, _capi.KPM_C128F):
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert cuda_lib.kpm_adjoint_forward(op.handle, R, M, ckpt, v.data_ptr(), mu.data_ptr(), s) == 0
        grad = torch.empty(n * L, dtype=torch.float64, device="cuda")
        assert cuda_lib.kpm_adjoint_backward_ex(op.handle, c.data_ptr(), grad.data_ptr(), dtype, s) == 0
        out.append(grad)
    scale = out[0].abs().max()
    assert scale > 0
    assert (out[0] - out[1]).abs().max() <= 16 * L * M * 2.0 ** -48 * scale
