"""The resident kernel's tallies, a copy per warp: the same as the
thread-per-electron kernel's, and no meeting point for its warps where they add
to them often (electrons of one or two events, channel counts)."""
import numpy as np
import pytest

from mcd import _lib, engine, tables

from _gpu_util import input_par

pytestmark = pytest.mark.gpu

RUNS = {
    "film": (dict(input_par("Si", 15000.0, 1000.0, 0.0, diffMFP=True, thickness=30.0)), 1000003),
    "film_cont": (dict(input_par("Cu", 15000.0, 1000.0, 70.0, mode="cont", bethe="JL", thickness=30.0)), 1000003),
    "channels": (dict(input_par("Si", 5000.0, 1000.0, 45.0)), 152001),
}


def median_us(p, n, block):
    import torch
    mat, tabs = _lib.material(p["material"]), None
    sim = engine.make_sim(p, n, 3, tally_flags=_lib.TALLY_CHANNELS)
    if sim.mode == _lib.MODE_DS:
        tabs = tables.ds_tables(mat, p["E0"], p["Emin"], p["Wc"], p["tol_E"], p["tol_W"])
        engine.use_sigma_table(sim, mat)
    bufs = engine.RunBuffers(n, _lib.FP32, True)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    times = []
    for _ in range(9):
        bufs.zero()
        ev[0].record()
        engine.launch(sim, mat, tabs, bufs, block)
        ev[1].record()
        torch.cuda.synchronize()
        times.append(1e3 * ev[0].elapsed_time(ev[1]))
    return float(np.median(times[2:])), engine.collect(bufs)


@pytest.mark.parametrize("name", list(RUNS))
def test_no_slower_than_a_thread_per_electron(name):
    (auto, a), (plain, b) = (median_us(*RUNS[name], block) for block in (0, 128))
    for k, v in a.tally.items():
        assert np.array_equal(v, b.tally[k]) or (k.startswith("sum_") and abs(v - b.tally[k]) <= 1e-9 * abs(v)), k
    assert sum(a.tally["channel"]) == a.tally["events"]
    assert auto < 1.3 * plain, (auto, plain)   # one copy for all warps: 6.0, 6.8 and 2.2 times
