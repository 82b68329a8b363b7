"""Channel counts: only the channels other than Rutherford are counted event by
event, so every count is checked against the events themselves, on the plain,
small-run and batched kernels, and members of a batch that do not ask for
counts keep theirs at zero."""
import numpy as np
import pytest

from mcd import _lib, engine

from _gpu_util import input_par

pytestmark = pytest.mark.gpu

CASES = {
    "si_film": dict(input_par("Si", 15000.0, 1000.0, 0.0, diffMFP=True, thickness=3000.0)),
    "au": dict(input_par("Au", 8000.0, 1000.0, 45.0)),
    "cu_cont": dict(input_par("Cu", 10000.0, 1000.0, 70.0, mode="cont", bethe="JL")),
}


def counted(p, n, **kw):
    r = engine.run(p, num_el=n, seed=4, ring_capacity=n * 1500, electrons=False, block_size=32, **kw)
    return np.bincount(r.events["step_chan"] & 31, minlength=_lib.MAX_CHANNELS)[:_lib.MAX_CHANNELS]


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("precision,block", [("fp32", 0), ("fp32", 64), ("fp64", 0), ("fp64", 8)])
def test_run_counts(name, precision, block):
    p, n = CASES[name], 301
    g = engine.run(p, num_el=n, seed=4, tally_channels=True, precision=precision, block_size=block)
    want = counted(p, n, precision=precision)
    assert np.array_equal(g.tally["channel"], want)
    assert int(want.sum()) == g.tally["events"]


def test_batch_counts_only_where_asked():
    names = list(CASES)
    b = engine.Batch([dict(CASES[k], num_el=301) for k in names], seed=4)
    b.structs[1].tally_flags = b.structs[2].tally_flags = _lib.TALLY_CHANNELS
    for k, s in enumerate(b.structs):
        s.sim_id = 0
        b._sims_arr[k] = s
    b.prepare()
    t, _ = b.run(_lib.Tune(128, 0, 1, 2, 0))   # cross sections per event, as the plain run
    assert not t[0]["channel"].any()
    for k in (1, 2):
        assert np.array_equal(t[k]["channel"], counted(CASES[names[k]], 301))
