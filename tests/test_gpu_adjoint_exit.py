"""The exit energy's gradient: the derivative carried along by the forward pass
and its product with dL/dE_exit over the backscattered electrons, at the edges
of the blocks and of the grid, for every Bethe law, and with electrons that
outran the checkpoint slots."""
import numpy as np
import pytest

from mcd import _lib
from mcd.adjoint import ExitEnergyModel
from _gpu_util import input_par

pytestmark = pytest.mark.gpu

NB, SIGMA = 64, 50.0


def model(n, precision, bethe="classical", species="Al", **kw):
    return ExitEnergyModel(input_par(species, 15000.0, 1000.0, 60.0, mode="cont", bethe=bethe), n, seed=9, nbins=NB,
                           sigma=SIGMA, precision=precision, **kw)


@pytest.mark.parametrize("bethe", ["classical", "JL", "explicit"])
@pytest.mark.parametrize("n", [1, 31, 257, 5000])
def test_equals_difference_along_frozen_sequence(n, bethe):
    """Per electron and unit weight a central difference at h = 1e-6 truncates
    to h^2/6 |K'''| |q'|^3 <= 1e-12/6 * 1.4 * (5e3/50)^3 < 1e-6 per bin in reach
    (about five, weights below 4), and rounds to 64 * 4 * 1e-16 / h < 1e-7; the
    gradient's terms are of order 10."""
    m = model(n, "fp64", bethe)
    _, _, nb = m.forward(1.1, 1.0)
    g = np.random.default_rng(n).uniform(-4.0, 4.0, NB)
    dJ, dn = m.backward(g, 0.0)
    h = 1e-6
    fd = (g @ (m.chain(1.1 + h)[0] - m.chain(1.1 - h)[0])) / (2.0 * h)
    # chain's J_scale is the multiplier itself, as the gradient's parameter is
    assert abs(dJ - fd) <= 1e-4 * max(nb, 1.0) / n
    assert dn == 0.0


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 320001])   # 320001: more than one trip of the grid
def test_product_over_electrons(n, precision):
    """Against NumPy from the pass's own inputs.  FP32: a bin's distance d is
    off by two roundings of an energy (2e-3 eV), its derivative by up to
    2e-3 / sigma^2 and the exponential's few 1e-6 / sigma besides."""
    m = model(n, precision)
    m.forward()
    r = np.random.default_rng(n)
    g, gs = r.uniform(-1.0, 1.0, NB), r.uniform(0.0, 1e-3)
    got, dn = m.backward(g, gs)
    ks = m.kstar.cpu().numpy()
    q, e = m.E_exit.cpu().numpy()[ks > 0].astype(float), m.ckpt[0].cpu().numpy()[ks > 0].astype(float)
    lo, w = m.hist.lo, (m.hist.hi - m.hist.lo) / NB
    d = q[:, None] - (lo + (np.arange(NB) + 0.5) * w)
    K = np.where(abs(d) <= 9.0 * SIGMA, np.exp(-d * d / (2.0 * SIGMA ** 2)), 0.0)
    lam = (K * -d / SIGMA ** 2) @ g / n + gs
    per_bin = 2.5e-3 / SIGMA ** 2 if precision == "fp32" else 1e-12
    # bins beyond 8 sigma are left out: 9 e^-32 / sigma each
    tol = (abs(e).sum() * (6 * per_bin + NB * 2e-13 / SIGMA)) / n + abs(lam * e).sum() * \
        (4e-7 if precision == "fp32" else 1e-13)
    assert abs(got - (lam * e).sum()) <= tol
    assert dn == 0.0


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_electrons_beyond_the_slots_carry_nothing(precision):
    n = 20000
    short, full = model(n, precision, species="Au", max_ckpt=1), model(n, precision, species="Au")
    short.launch_forward()
    full.forward()
    assert int(short.status.cpu()[0]) & _lib.FLAG_CKPT
    assert (short.kstar == full.kstar).all() and (full.kstar > 64).any()
    full.kstar[full.kstar > 64] = -1
    g = np.random.default_rng(0).standard_normal(NB)
    a, b = short.backward(g, 1.0)[0], full.backward(g, 1.0)[0]
    assert a == pytest.approx(b, rel=1e-9)   # FP64 sums in another order


def test_gradient_that_is_not_finite_shows():
    m = model(2000, "fp32")
    m.forward()
    dJ, dn = m.backward(np.full(NB, np.nan), 0.0)
    assert np.isnan(dJ) and np.isnan(dn)
