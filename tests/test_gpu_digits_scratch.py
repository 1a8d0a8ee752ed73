"""The table contractions keep no scratch in the handle: a recorded graph of them replays after the handle's
own buffers were freed and grown, calls of one handle on two streams do not disturb each other, and a
workspace that is missing, short or misaligned is refused."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_recorded_moments_after_the_handle_has_grown(cuda_lib):
    import torch

    from minijclsquant_gb300 import adjoint, device

    plan = adjoint.KuboPlan(12, 11, 70, R=2, n_energies=8)
    want = plan.mu_nm()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = plan.mu_nm()
    v = torch.ones((8, plan.n), dtype=torch.complex128, device="cuda")
    device.cheb_moments(plan.op_h, 3000, v)  # larger buffers of the same handle
    held = [torch.full((1 << 22,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(8)]
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)  # the same sums: recorded tables are equal up to the sign of a zero
    assert cuda_lib.kpm_ell_check(plan.op_h.handle, None) == 0 and len(held) == 8


@pytest.mark.parametrize("M,n", [(33, 900), (128, 5000)])
def test_two_streams(cuda_lib, M, n):
    import torch

    from minijclsquant_gb300.device import DeviceELL

    h = DeviceELL(np.full(n, 0.5 + 0j), np.arange(n, dtype=np.int32), 1)
    rng = np.random.default_rng(M)
    sets = []
    for _ in range(2):
        t = [torch.from_numpy(rng.standard_normal((M, n)) + 1j * rng.standard_normal((M, n))).cuda() for _ in range(2)]
        sets.append(t + [torch.from_numpy(rng.standard_normal((M, M))).cuda()])

    def run(u, w, c):
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        mu, q = torch.empty((M, M), dtype=torch.complex128, device="cuda"), torch.empty_like(u)
        assert cuda_lib.kpm_table_gram(h.handle, M, u.data_ptr(), w.data_ptr(), 0, mu.data_ptr(), s) == 0
        assert cuda_lib.kpm_table_mix(h.handle, M, c.data_ptr(), u.data_ptr(), q.data_ptr(), s) == 0
        return mu, q

    want = [run(*t) for t in sets]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        got = []
        for t, st in zip(sets, streams):
            with torch.cuda.stream(st):
                got.append(run(*t))
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for x, y in zip(got, want) for a, b in zip(x, y))
    assert cuda_lib.kpm_ell_check(h.handle, None) == 0


def test_workspace_is_checked(cuda_lib):
    import torch

    from minijclsquant_gb300 import _capi
    from minijclsquant_gb300.device import DeviceELL

    M, n = 9, 100
    h = DeviceELL(np.full(n, 0.5 + 0j), np.arange(n, dtype=np.int32), 1)
    u = torch.ones((M, n), dtype=torch.complex128, device="cuda")
    c = torch.ones((M, M), dtype=torch.float64, device="cuda")
    mu, q = torch.empty((M, M), dtype=torch.complex128, device="cuda"), torch.empty_like(u)
    need = cuda_lib.kpm_table_work_bytes(h.handle, M)
    assert need > 0 and cuda_lib.kpm_table_work_bytes(None, M) == 0
    work = torch.empty(need + 16, dtype=torch.uint8, device="cuda")
    for ptr, size in ((None, need), (work.data_ptr(), need - 1), (work.data_ptr() + 16, need)):
        for st in (cuda_lib.kpm_table_gram_work(h.handle, M, u.data_ptr(), u.data_ptr(), 0, mu.data_ptr(), ptr, size, None),
                   cuda_lib.kpm_table_mix_work(h.handle, M, c.data_ptr(), u.data_ptr(), q.data_ptr(), ptr, size, None)):
            assert st == _capi.KPM_ERR_INVALID_ARG
    assert cuda_lib.kpm_table_gram_work(h.handle, M, u.data_ptr(), u.data_ptr(), 0, mu.data_ptr(), work.data_ptr(), need,
                                        None) == 0
    assert cuda_lib.kpm_table_mix_work(h.handle, M, c.data_ptr(), u.data_ptr(), q.data_ptr(), work.data_ptr(), need,
                                       None) == 0
    torch.cuda.synchronize()
    assert torch.equal(mu, torch.full_like(mu, n)) and torch.equal(q, torch.full_like(q, M))
