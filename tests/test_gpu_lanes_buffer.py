"""The small-run kernel's buffer of values computed ahead, in the continuous
model with every event recorded: there lane 0 alone appends the records, and no
vote or shuffle of the event meets the lanes, so only the barrier before the
buffer's older half is overwritten keeps its values for a lane that lags.
Trajectories of many times 32 events (each half overwritten many times),
compared with the thread-per-electron kernel record by record."""
import numpy as np
import pytest

from mcd import engine

from _gpu_util import input_par

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 37, 152, 11 * 152])   # all with 32 lanes per electron
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_continuous_records_equal_plain(n, precision):
    p = dict(input_par("Au", 25000.0, 1000.0, 0.0, mode="cont", bethe="JL"))
    a, b = (engine.run(p, num_el=n, seed=11, precision=precision, ring_capacity=1500 * n + 4096, block_size=k)
            for k in (0, 64))
    assert a.events_total == b.events_total <= 1500 * n + 4096
    assert int(a.electrons["n_events"].max()) > 8 * 32
    for f in a.electrons:
        assert np.array_equal(a.electrons[f], b.electrons[f]), f
    key = lambda e: e[np.lexsort((e["step_chan"], e["electron"]))].tobytes()  # noqa: E731
    assert key(a.events) == key(b.events)
