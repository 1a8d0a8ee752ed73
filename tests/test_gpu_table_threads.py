"""Vector tables of one operator from several host threads, each on a stream of its own: the calls share the
handle's words for the one-launch form and must take turns."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tables_from_threads(cuda_lib):
    import torch

    from minijclsquant_gb300 import device, lattice

    g = lattice.honeycomb_device(60, 50, W=1.0, seed=1)
    n, M, threads = g.n, 40, 4
    s_op = device.DeviceELL(1j * g.data_kpm, g.indices, g.len_row)
    rng = np.random.default_rng(0)
    z = [torch.from_numpy(rng.normal(size=(M, n)) + 1j * rng.normal(size=(M, n))).cuda() for _ in range(threads)]

    def run(x, out, stream):
        tab, stab, lam = out
        status = cuda_lib.kpm_cheb_table(g.op.handle, s_op.handle, M, x.data_ptr(), tab.data_ptr(), stab.data_ptr(), stream)
        return status or cuda_lib.kpm_cheb_clenshaw_table(g.op.handle, s_op.handle, M, x.data_ptr(), lam.data_ptr(), stream)

    outs = lambda: [tuple(torch.empty_like(z[0]) for _ in range(3)) for _ in range(threads)]  # noqa: E731
    want, got = outs(), outs()
    for x, o in zip(z, want):
        assert run(x, o, None) == 0
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(threads)]
    status = [0] * threads
    start = threading.Barrier(threads)

    def work(i):
        start.wait()
        for _ in range(25):
            status[i] |= run(z[i], got[i], ctypes.c_void_p(streams[i].cuda_stream))

    pool = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    torch.cuda.synchronize()
    assert status == [0] * threads
    assert cuda_lib.kpm_ell_check(g.op.handle, None) == 0
    for a, b in zip(want, got):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
