"""The automatic choice of an FP32 run's kernel is not slower than a
thread per electron in blocks of 128 (or less, where those leave SMs idle), at
sizes on both sides of its lines and where trajectories are short."""
import numpy as np
import pytest

from mcd import _lib, engine, tables

from _gpu_util import input_par

pytestmark = pytest.mark.gpu

SMS = 152
RUNS = {
    "al_5": input_par("Al", 5000.0, 500.0, 60.0, mode="cont", bethe="JL"),
    "si_10": input_par("Si", 10000.0, 1000.0, 80.0, mode="cont", bethe="JL"),
    "cu_10": input_par("Cu", 10000.0, 1000.0, 60.0, mode="cont", bethe="JL"),
    "au_10": input_par("Au", 10000.0, 1000.0, 0.0, mode="cont", bethe="JL"),
    "thin": input_par("Cu", 15000.0, 1000.0, 20.0, thickness=100.0),
    "film": input_par("Si", 30000.0, 1000.0, 75.0, mode="cont", bethe="JL", thickness=1000.0),
}


def median_us(p, n, block):
    import torch
    mat = _lib.material(p["material"])
    sim = engine.make_sim(p, n, 3)
    tabs = None
    if sim.mode == _lib.MODE_DS:
        tabs = tables.ds_tables(mat, p["E0"], p["Emin"], p["Wc"], p["tol_E"], p["tol_W"])
    bufs = engine.RunBuffers(n, _lib.FP32, True)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    times = []
    for _ in range(24):
        bufs.zero()
        ev[0].record()
        engine.launch(sim, mat, tabs, bufs, block)
        ev[1].record()
        torch.cuda.synchronize()
        times.append(1e3 * ev[0].elapsed_time(ev[1]))
    return float(np.median(times[4:]))


@pytest.mark.parametrize("per_sm", [33, 240, 500, 900])
@pytest.mark.parametrize("name", list(RUNS))
def test_not_slower_than_independent_threads(name, per_sm):
    n, block = per_sm * SMS, 128
    while block > 8 and -(-n // block) < SMS:
        block //= 2
    for _ in range(4):   # tens of us: one pair of medians can be off by a tenth
        auto, plain = median_us(RUNS[name], n, 0), median_us(RUNS[name], n, block)
        if auto <= 1.08 * plain:
            return
    pytest.fail("%.1f us, independent threads %.1f" % (auto, plain))
