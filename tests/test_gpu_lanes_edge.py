"""Beam energies that FP32 rounds to Emin: an electron then ends with its first
event, whatever the event, in every kernel that an FP32 run can take."""
import numpy as np
import pytest

from mcd import _lib, engine, tables

from _gpu_util import input_par

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("n", [1, 5 * SMS, 25 * SMS, 40 * SMS, 70 * SMS])   # 32, 16, 8 lanes and one per electron
@pytest.mark.parametrize("quirks", [0, _lib.QUIRKS_REFERENCE])
@pytest.mark.parametrize("film", [False, True])
@pytest.mark.parametrize("tabulated", [False, True])
def test_beam_at_the_cutoff(n, quirks, film, tabulated):
    kw = dict(diffMFP=True, thickness=3000.0) if film else {}
    p = dict(input_par("Si", 1000.00001, 1000.0, 20.0, **kw))
    assert np.float32(p["E0"]) == np.float32(p["Emin"]) and p["E0"] > p["Emin"]
    tabs = tables.ds_tables(_lib.material("Si"), 5000.0, 1000.0, 100.0, 1e-3, 1e-3)
    a, b = (engine.run(p, num_el=n, seed=9, tables=tabs, quirks=quirks, tabulated=tabulated, tally_channels=True,
                       block_size=k) for k in (0, 64))
    assert a.tally["events"] == n
    for f in a.electrons:
        assert np.array_equal(a.electrons[f], b.electrons[f]), f
    for k, v in a.tally.items():
        assert np.array_equal(v, b.tally[k]) or (k.startswith("sum_") and abs(v - b.tally[k]) <= 1e-12 * abs(v)), k
