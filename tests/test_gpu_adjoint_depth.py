"""The deepest z's gradient, whose backward pass sorts the backscattered
electrons of a block's range by the length of their sequences: at the edges of
warps, blocks and ranges (1024, 2048 and 4096 electrons, by the size of the run),
with electrons that outran the checkpoint slots."""
import numpy as np
import pytest

from mcd import _lib
from mcd.adjoint import ExitEnergyModel
from _gpu_util import input_par

pytestmark = pytest.mark.gpu

NB, SIGMA = 64, 300.0


def model(n, precision, species="Al", **kw):
    return ExitEnergyModel(input_par(species, 15000.0, 1000.0, 60.0, mode="cont", bethe="classical"), n, seed=5,
                           nbins=NB, sigma=SIGMA, lo=0.0, hi=20000.0, precision=precision, quantity="max_depth", **kw)


# the last two: the first sizes of a range of 2048 and of 4096 electrons on 152 SMs
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [1, 33, 1023, 1025, 5000, 155649, 311297])
def test_density_gradient_counts_every_electron_once(n, precision):
    """Z is proportional to 1/n_scale, so dL/dn = -sum over electrons of
    dL/dZ Z / N: NumPy's sum from the pass's own Z.  The sweep sums some tens to
    hundreds of positive and negative terms g s d_z per electron: within
    1e-4 (FP32) or 1e-12 (FP64) of sum |dL/dZ| Z, plus, in FP32, the rounding of
    the bins' distances (2e-3 A at most, in g 2e-3 / sigma^2 per bin in reach,
    at most 16)."""
    m = model(n, precision)
    m.forward()
    r = np.random.default_rng(n)
    g, gs = r.uniform(-1.0, 1.0, NB), r.uniform(0.0, 1e-3)
    _, dn = m.backward(g, gs)
    ks = m.kstar.cpu().numpy()
    Z = m.E_exit.cpu().numpy()[ks > 0].astype(float)
    lo, w = m.hist.lo, (m.hist.hi - m.hist.lo) / NB
    d = Z[:, None] - (lo + (np.arange(NB) + 0.5) * w)
    K = np.where(abs(d) <= 9.0 * SIGMA, np.exp(-d * d / (2.0 * SIGMA ** 2)), 0.0)
    lam = (K * -d / SIGMA ** 2) @ g / n + gs
    rel, per_bin = (1e-4, 2e-3 / SIGMA ** 2) if precision == "fp32" else (1e-12, 1e-14)
    tol = rel * abs(lam * Z).sum() + (16 * per_bin + NB * 2e-13 / SIGMA) * Z.sum() / n
    assert abs(dn + (lam * Z).sum()) <= tol


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_electrons_beyond_the_slots_carry_nothing(precision):
    n = 20000
    short, full = model(n, precision, species="Au", max_ckpt=1), model(n, precision, species="Au")
    short.launch_forward()
    full.forward()
    assert int(short.status.cpu()[0]) & _lib.FLAG_CKPT
    full.kstar[full.kstar > 64] = -1
    g = np.random.default_rng(0).standard_normal(NB)
    a, b = short.backward(g, 1.0), full.backward(g, 1.0)
    assert a == pytest.approx(b, rel=1e-9)   # the same electrons' FP64 sums in another order
