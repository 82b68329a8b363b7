"""The run-down list of a batched launch is apart from the workspace: a batch's
workspace holds nothing that grows with the launch, a list no more than its
electrons, and the chunks of a stream share one."""
import numpy as np
import pytest

from mcd import _lib, engine, stream

from _gpu_util import input_par


def test_sizes():
    L = _lib.lib()
    for n in (1, 6, 64, 256):   # the upload and a table slot (4096 x 12 floats) per simulation
        assert L.mcd_batch_workspace_bytes(n) == L.mcd_batch_upload_bytes(n) + n * 4 * 4096 * 12
    assert [L.mcd_batch_list_bytes(n) for n in (-1, 0, 1, 1000, 2 ** 18, 2 ** 40)] == [0, 0, 68, 68000, 68 << 18, 68 << 18]


@pytest.mark.gpu
def test_stream_of_many_chunks_holds_one_list():
    import torch
    p = dict(input_par("Si", 5000.0, 1000.0, 0.0), num_el=6000)
    small = stream.EventStream(dict(p, num_el=50), chunk=50, seed=2, ring_events=200000, piece_bytes=1 << 20)   # the tables
    before = torch.cuda.memory_allocated()
    s = stream.EventStream(p, chunk=50, seed=2, ring_events=200000, piece_bytes=1 << 20)
    used = torch.cuda.memory_allocated() - before
    # per chunk: the workspace, the tally and the status, each rounded up to 512
    per = _lib.lib().mcd_batch_workspace_bytes(1) + 256 + 4096 + 3 * 512
    assert s.nchunks == 120
    assert used <= 120 * per + 2 * 200000 * s.rec_bytes + 50 * 68 + (4 << 20)
    got = s.run()
    ref, _ = engine.Batch([p], seed=2).run()
    for k in ("bks", "abs", "events"):
        assert sum(t[k] for t in got["tallies"]) == ref[0][k]
    assert small.run()["events"] > 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 33, 3000, 400000])
def test_endings_agree(n):
    """With its list, with none and with one too small."""
    sims = [dict(input_par(m, 5000.0, 1000.0, 45.0), num_el=n // (k + 1) + 1) for k, m in enumerate(("Au", "Si"))]
    ref, st = engine.Batch(sims, seed=4, electrons=False).run()
    import torch
    for size in (0, 68 * 20):
        got, st2 = engine.Batch(sims, seed=4, scratch=torch.empty(size, dtype=torch.uint8, device="cuda")).run()
        assert st2 == st
        for a, b in zip(got, ref):
            for k, v in a.items():
                same = abs(v - b[k]) <= 1e-9 * abs(v) if k.startswith("sum_") else np.array_equal(v, b[k])
                assert same, k
