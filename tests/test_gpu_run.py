"""The resident kernel of large FP32 runs and the run-down kernel of batches
against the thread-per-electron kernel: rows, tallies and events bit for bit at
the sizes where the block shape, the refill and the compaction change."""
import numpy as np
import pytest

from mcd import _lib, engine

from _gpu_util import input_par
from test_gpu_lanes import SMS, same

pytestmark = pytest.mark.gpu

RUNS = {
    "au": dict(input_par("Au", 4000.0, 500.0, 45.0, Wc=50.0)),
    "film": dict(input_par("Si", 9000.0, 1000.0, 20.0, diffMFP=True, thickness=2500.0)),
    "limit": dict(input_par("Si", 5000.0, 1000.0, 0.0), maxScatt=150),
    "cont": dict(input_par("Cu", 10000.0, 1000.0, 70.0, mode="cont", bethe="JL")),
}
# one warp per SM partly filled, one wave of 512, the change to 896, one wave of
# them and more than one
SIZES = [58 * SMS, 70 * SMS + 1, 257 * SMS - 3, 512 * SMS, 512 * SMS + 1, 896 * SMS, 896 * SMS + 1, 2300 * SMS + 1]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("name", list(RUNS))
@pytest.mark.parametrize("tabulated", [False, True])
def test_rows_equal_plain(name, n, tabulated):
    kw = dict(num_el=n, seed=n, tabulated=tabulated, tally_channels=True, first_electron=2 ** 32 - 1000)
    same(engine.run(RUNS[name], **kw), engine.run(RUNS[name], block_size=128, **kw))


@pytest.mark.parametrize("n", [70 * SMS + 1, 600 * SMS])
@pytest.mark.parametrize("name", ["film", "au", "cont"])
def test_events_equal_plain(name, n):
    p, cap = RUNS[name], 300 * n
    fields = _lib.EV_E | _lib.EV_C2 | _lib.EV_PACKED_HEAD   # the unpacked form needs each electron's order kept
    a, b = (engine.run(p, num_el=n, seed=5, ring_capacity=cap, ring_fields=fields, block_size=k) for k in (0, 128))
    same(a, b)
    assert a.events_total == b.events_total <= cap
    assert a.events.tobytes() == b.events.tobytes()


@pytest.mark.parametrize("tune", [(256, 0, 1, 2, 0), (576, 0, 1, 3, 0), (1024, 0, 32, 2, 0), (32, 1, 16, 2, 0)])
@pytest.mark.parametrize("scale", [1, 40])
def test_batches_equal_plain(tune, scale):
    # scale 1: fewer electrons than lanes (all listed at once); 40: several per lane
    sims = [dict(p, num_el=k * scale) for p, k in zip(RUNS.values(), (1500, 2501, 777, 1201))]
    b = engine.Batch(sims, seed=12, tally_channels=True, electrons=True)
    tallies, status = b.run(_lib.Tune(*tune))
    st = 0
    for k, p in enumerate(sims):
        mat = _lib.material(p["material"])
        sim = engine.make_sim(p, p["num_el"], 12, sim_id=k, tally_flags=_lib.TALLY_CHANNELS)
        tabs = (None if p["mode"] == "cont" else
                engine.ds_tables(mat, *(p[f] for f in ("E0", "Emin", "Wc", "tol_E", "tol_W"))))
        bufs = engine.RunBuffers(p["num_el"])
        engine.launch(sim, mat, tabs, bufs, 128)
        r = engine.collect(bufs)
        st |= r.status
        same(engine.RunResult(tallies[k], r.status, b.electrons(k)), r)
    assert status == st


def test_batch_events_keep_their_order():
    sims = [dict(RUNS["au"], num_el=3000)]
    fields = _lib.EV_E | _lib.EV_PACKED_HEAD
    b = engine.Batch(sims, seed=3)
    _, _, ev, total = b.run_events(3000 * 400, fields, _lib.Tune(128, 0, 1, 2, 0))
    r = engine.run(dict(RUNS["au"]), num_el=3000, seed=3, ring_capacity=3000 * 400, ring_fields=fields, block_size=64)
    assert total == r.events_total
    assert ev.tobytes() == r.events.tobytes()


@pytest.mark.parametrize("n", [1, 8191, 8192, 20001])
@pytest.mark.parametrize("precision", [_lib.FP32, _lib.FP64])
def test_rows_read_back_are_the_device_arrays(n, precision):
    p = dict(RUNS["cont"], maxScatt=20)
    bufs = engine.RunBuffers(n, precision, ring_capacity=30 * n)
    bufs.zero()
    engine.launch(engine.make_sim(p, n, 1, precision=precision), _lib.material(p["material"]), None, bufs)
    r = engine.collect(bufs)
    el = {k: v.cpu().numpy() for k, v in bufs.el.items()}
    for k in ("outcome", "flags", "final_E", "max_z", "n_events"):
        assert np.array_equal(r.electrons[k], el[k]), k
    for k in ("dir", "last_pos"):
        assert r.electrons[k].shape == (n, 3) and r.electrons[k].flags.c_contiguous
        assert np.array_equal(r.electrons[k], el[k].reshape(3, n).T), k
    assert r.tally["events"] == int(el["n_events"].sum()) == r.events_total == int(bufs.cursor.item())
    t = _lib.Tally.from_buffer_copy(bufs.tally.cpu().numpy().tobytes())
    assert list(t.channel) == r.tally["channel"].tolist() and t.sum_E_bks == r.tally["sum_E_bks"]
    assert list(t.hist_E) == r.tally["hist_E"].tolist() and list(t.hist_T) == r.tally["hist_T"].tolist()
