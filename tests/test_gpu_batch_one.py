"""Batches of one simulation, whose run-down kernel keeps the simulation's
constants in registers: rows, tallies and events equal the thread-per-electron
kernel's bit for bit, below and above a launch's lanes."""
import pytest

from mcd import _lib, engine

from test_gpu_lanes import SMS, same
from test_gpu_run import RUNS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("n", [1, 33, 90 * SMS, 1100 * SMS + 1])
@pytest.mark.parametrize("name", list(RUNS))
def test_rows_equal_plain(name, n, channels):
    b = engine.Batch([dict(RUNS[name], num_el=n)], seed=8, tally_channels=channels, electrons=True)
    tallies, status = b.run(_lib.Tune(256, 0, 1, 2, 0))   # cross sections per event, as the plain run
    r = engine.run(RUNS[name], num_el=n, seed=8, tabulated=False, tally_channels=channels, block_size=128)
    same(engine.RunResult(tallies[0], status, b.electrons(0)), r)


@pytest.mark.parametrize("n", [33, 90 * SMS])
@pytest.mark.parametrize("name", ["film", "cont"])
def test_events_equal_plain(name, n):
    cap, fields = 300 * n, _lib.EV_E | _lib.EV_C2 | _lib.EV_PACKED_HEAD
    b = engine.Batch([dict(RUNS[name], num_el=n)], seed=5)
    _, _, ev, total = b.run_events(cap, fields, _lib.Tune(128, 0, 1, 2, 0))
    r = engine.run(RUNS[name], num_el=n, seed=5, tabulated=False, ring_capacity=cap, ring_fields=fields, block_size=128)
    assert total == r.events_total <= cap
    assert ev.tobytes() == r.events.tobytes()
