"""The per-electron Philox constants at electron indices around a 32-bit word
boundary: trajectories follow the oracle's own counters, and every electron's
row lands at its index (the batched kernel recovers it from the constants)."""
import numpy as np
import pytest

import coracle
import mcd_oracle as O
from mcd import _lib, engine

from _gpu_util import input_par

pytestmark = pytest.mark.gpu

FIRSTS = [0, 1, 2 ** 32 - 5, 2 ** 32, 7 * 2 ** 32 - 1, (5 << 40) + 3, 2 ** 63 + 11]


@pytest.mark.parametrize("first", FIRSTS)
@pytest.mark.parametrize("seed", [3, 2 ** 64 - 1])
def test_continuous_rows_follow_the_oracle(first, seed):
    p = input_par("Al", 5000.0, 1000.0, 45.0, mode="cont", bethe="classical")
    n = 40
    g = engine.run(p, num_el=n, seed=seed, first_electron=first, precision="fp64")
    c = coracle.run(O.Material("Al"), p["E0"], p["Emin"], p["s_tilt"], n, seed=seed, first=first, mode="cont")
    assert np.array_equal(g.electrons["n_events"], c["n_events"])
    assert np.array_equal(g.electrons["outcome"], c["outcome"])


@pytest.mark.parametrize("first", FIRSTS)
def test_batched_rows_equal_plain(first):
    p = dict(input_par("Si", 5000.0, 1000.0, 20.0), num_el=97)
    q = dict(input_par("Cu", 6000.0, 1000.0, 0.0, mode="cont", bethe="JL"), num_el=61)
    b = engine.Batch([p, q], seed=9, first_electron=first, electrons=True)
    b.run(_lib.Tune(64, 0, 1, 2, 0))    # cross sections per event, as the plain launch below
    for k, x in enumerate((p, q)):
        mat = _lib.material(x["material"])
        sim = engine.make_sim(x, x["num_el"], 9, first, sim_id=k)
        bufs = engine.RunBuffers(x["num_el"])
        tabs = engine.ds_tables(mat, *(x[f] for f in ("E0", "Emin", "Wc", "tol_E", "tol_W"))) if k == 0 else None
        engine.launch(sim, mat, tabs, bufs, 32)
        r, e = engine.collect(bufs).electrons, b.electrons(k)
        for f in r:
            assert np.array_equal(r[f], e[f]), f
