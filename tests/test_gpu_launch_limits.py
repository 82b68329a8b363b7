"""Launches that need more shared memory than a block has by default, of unlike
sizes and from two threads at once: one thread's launch may not take back the
limit that another's has just asked for."""
import ctypes as C
import threading

import numpy as np
import pytest

from mcd import _lib, engine

from _gpu_util import input_par

pytestmark = pytest.mark.gpu


def both(calls, times):
    codes = [set(), set()]
    gate = threading.Barrier(2)

    def loop(k):
        gate.wait()
        for _ in range(times):
            codes[k].add(calls[k]())

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return codes


def test_tables_of_unlike_widths_from_two_threads():
    import torch
    mat = _lib.material("Si")

    def fill(nW):
        Ws = torch.from_numpy(np.geomspace(100.0, 4000.0, nW, dtype=np.float32)).cuda()
        Es = torch.from_numpy(np.linspace(1000.0, 9000.0, 8, dtype=np.float32)).cuda()
        cdf = torch.empty((8, nW - 1), dtype=torch.float32, device="cuda")
        st = torch.cuda.Stream()
        torch.cuda.synchronize()
        f = lambda: _lib.lib().mcd_build_table(0, C.byref(mat), 0, 8, nW, Es.data_ptr(), Ws.data_ptr(),  # noqa: E731
                                               cdf.data_ptr(), None, None, None, st.cuda_stream)
        return f, (Ws, Es, cdf, st)

    fills = [fill(nW) for nW in (480, 1000)]   # 51 and 104 KB
    codes = both([f for f, _ in fills], 5000)
    torch.cuda.synchronize()
    assert codes == [{_lib.OK}, {_lib.OK}]


def test_batches_of_unlike_sizes_from_two_threads():
    import torch

    def batch(n):
        b = engine.Batch([dict(input_par("Al", 5000.0, 1000.0, 0.0), num_el=1)] * n, seed=1)
        st, tune = torch.cuda.Stream(), _lib.Tune(256, 0, 1, 0, 0)
        torch.cuda.synchronize()
        f = lambda: _lib.lib().mcd_run_batched(b.ws_ptr, b.n, b.tallies.data_ptr(), C.byref(tune),  # noqa: E731
                                               b.status.data_ptr(), st.cuda_stream)
        return f, (b, st, tune)

    batches = [batch(n) for n in (80, 120)]
    codes = both([f for f, _ in batches], 2000)
    torch.cuda.synchronize()
    assert codes == [{_lib.OK}, {_lib.OK}]
