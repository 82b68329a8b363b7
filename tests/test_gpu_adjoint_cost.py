"""What carrying the exit energy's derivative along adds to an FP64 forward
pass, against the depth's forward pass, which carries none: less than a fifth
for the laws that have a J (four divisions an event took a quarter), nothing for
the explicit one."""
import numpy as np
import pytest

from mcd.adjoint import ExitEnergyModel

from _gpu_util import input_par

pytestmark = pytest.mark.gpu


def forward_us(bethe, **kw):
    import torch
    m = ExitEnergyModel(input_par("Al", 15000.0, 1000.0, 70.0, mode="cont", bethe=bethe), 30000, seed=1,
                        precision="fp64", **kw)
    m.forward()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    times = []
    for _ in range(9):
        ev[0].record()
        m.launch_forward()
        ev[1].record()
        torch.cuda.synchronize()
        times.append(1e3 * ev[0].elapsed_time(ev[1]))
    return float(np.median(times[2:]))


@pytest.mark.parametrize("bethe, most", [("classical", 1.2), ("JL", 1.2), ("explicit", 1.07)])
def test_derivative_along_the_forward_pass(bethe, most):
    for _ in range(3):
        exit_e, depth = forward_us(bethe), forward_us(bethe, quantity="max_depth", lo=0.0, hi=20000.0, sigma=300.0)
        if exit_e <= most * depth:
            return
    pytest.fail("%.0f us, without a derivative %.0f" % (exit_e, depth))
