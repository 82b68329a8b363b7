"""The small-run kernel (several lanes per electron) against the thread-per-
electron kernel: rows, tallies and event records bit for bit, at the run sizes
that select each group width, for both modes and precisions, with and without
the cross-section tables, in the diffracting film and at the event limit."""
import numpy as np
import pytest

from mcd import engine

from _gpu_util import input_par

pytestmark = pytest.mark.gpu

RUNS = {
    "si": dict(input_par("Si", 10000.0, 1000.0, 0.0)),
    "au": dict(input_par("Au", 8000.0, 500.0, 45.0, Wc=50.0)),
    "cu_low": dict(input_par("Cu", 5000.0, 150.0, 70.0)),          # below 2 Wc: a bent row, flagged cells
    "film": dict(input_par("Si", 15000.0, 1000.0, 20.0, diffMFP=True, thickness=3000.0)),
    "nigram": dict(input_par("Al", 6000.0, 1000.0, 0.0, elastic="Ruth_nigram")),
    "limit": dict(input_par("Si", 10000.0, 1000.0, 0.0), maxScatt=77),
    "cont": dict(input_par("Cu", 9000.0, 1000.0, 70.0, mode="cont", bethe="JL")),
    "cont_ex": dict(input_par("Al", 5000.0, 1000.0, 0.0, mode="cont", bethe="explicit"), maxScatt=150),
}
SMS = 152
# electrons per SM: below 3, 8, 16, 18, 20, 33, 34, 47 and 58 the group width changes
SIZES = [1, 2, 3, 31, 2 * SMS + 1, 4 * SMS, 9 * SMS + 5, 11 * SMS, 25 * SMS + 3, 40 * SMS + 7]


def same(a, b):
    for f in a.electrons:
        assert np.array_equal(a.electrons[f], b.electrons[f], equal_nan=a.electrons[f].dtype.kind == "f"), f
    for k, v in a.tally.items():
        if k.startswith("sum_"):
            assert abs(v - b.tally[k]) <= 1e-12 * abs(v)   # FP64 sums in another order
        else:
            assert np.array_equal(v, b.tally[k]), k
    assert a.status == b.status


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("name", list(RUNS))
@pytest.mark.parametrize("tabulated", [False, True])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_rows_equal_plain(name, n, tabulated, precision):
    p = RUNS[name]
    if precision == "fp64" and n > 12 * SMS:
        n = n // 3
    kw = dict(num_el=n, seed=n, precision=precision, tabulated=tabulated, tally_channels=True, first_electron=2 ** 32 - 7)
    same(engine.run(p, **kw), engine.run(p, block_size=64, **kw))


@pytest.mark.parametrize("n", [8 * SMS - 1, 8 * SMS, 16 * SMS - 1, 16 * SMS, 18 * SMS - 1, 18 * SMS, 47 * SMS - 1, 47 * SMS])
@pytest.mark.parametrize("name", ["si", "au", "film", "limit", "cont"])
def test_fp64_rows_equal_plain_at_the_widths(name, n):
    kw = dict(num_el=n, seed=n, precision="fp64", tabulated=True, tally_channels=True)
    same(engine.run(RUNS[name], **kw), engine.run(RUNS[name], block_size=64, **kw))


@pytest.mark.parametrize("n", [1, 37, 27 * SMS])
@pytest.mark.parametrize("name", ["si", "film", "cont"])
def test_events_equal_plain(name, n):
    p, cap = RUNS[name], 900 * n + 64
    a, b = (engine.run(p, num_el=n, seed=5, ring_capacity=cap, block_size=k, tabulated=True) for k in (0, 64))
    same(a, b)
    assert a.events_total == b.events_total <= cap
    key = lambda e: e[np.lexsort((e["step_chan"], e["electron"]))].tobytes()  # noqa: E731
    assert key(a.events) == key(b.events)
