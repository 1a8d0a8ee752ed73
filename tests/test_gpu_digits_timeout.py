"""A wait of the digit GEMM that runs out, for all of its warps or for one epilogue warp alone: the kernel
ends promptly, the status says so once, and the next product is right.  No copy is left in flight and
nothing faults (kpm_table_test_timeout)."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warp", [-1, 0, 3, 7])
def test_timeout_ends_the_kernel(cuda_lib, warp):
    import torch

    from minijclsquant_gb300 import _capi
    from minijclsquant_gb300.device import DeviceELL

    M, n = 5, 40
    h = DeviceELL(np.full(n, 0.5 + 0j), np.arange(n, dtype=np.int32), 1)
    assert cuda_lib.kpm_table_test_timeout(h.handle, 10, warp, None) == _capi.KPM_ERR_INVALID_ARG
    assert cuda_lib.kpm_table_test_timeout(h.handle, 20_000_000, 8, None) == _capi.KPM_ERR_INVALID_ARG
    t0 = time.perf_counter()
    assert cuda_lib.kpm_table_test_timeout(h.handle, 20_000_000, warp, None) == _capi.KPM_ERR_TIMEOUT
    assert time.perf_counter() - t0 < 5.0
    assert cuda_lib.kpm_ell_check(h.handle, None) == _capi.KPM_OK
    u = torch.ones((M, n), dtype=torch.complex128, device="cuda")
    mu = torch.empty((M, M), dtype=torch.complex128, device="cuda")
    assert cuda_lib.kpm_table_gram(h.handle, M, u.data_ptr(), u.data_ptr(), 0, mu.data_ptr(),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert torch.equal(mu, torch.full_like(mu, n))
