"""The soft-bin pass of the adjoint's forward on the quantities the forward left
per electron: against NumPy in FP64, and in FP32, whose weights are rounded in
their own way, against the per-thread bins of the frozen-sequence chain (the
same quantities, recomputed bit for bit).  Bin counts around the 32 lanes of a
warp and up to the largest, electron counts around a warp and a block."""
import numpy as np
import pytest

from mcd.adjoint import ExitEnergyModel

from _gpu_util import input_par

pytestmark = pytest.mark.gpu

P = input_par("Cu", 8000.0, 1000.0, 70.0, mode="cont", bethe="JL")


@pytest.mark.parametrize("nbins", [1, 31, 32, 33, 64, 65, 256])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 5000])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("quantity", ["exit_E", "max_depth"])
def test_bins(nbins, n, precision, quantity):
    kw = dict(lo=0.0, hi=3000.0, sigma=40.0) if quantity == "max_depth" else dict(sigma=60.0)
    m = ExitEnergyModel(P, n, seed=n, nbins=nbins, precision=precision, quantity=quantity, **kw)
    h, total, count = m.forward()
    q = m.E_exit.cpu().numpy().astype(np.float64)[m.kstar.cpu().numpy() >= 0]
    lo, hi, sigma = m.hist.lo, m.hist.hi, m.hist.sigma
    c = lo + (np.arange(nbins) + 0.5) * (hi - lo) / nbins
    want = np.exp(-(q[:, None] - c) ** 2 / (2.0 * sigma * sigma)).sum(axis=0) / n
    assert count == q.size
    # beyond 8 sigma (1e-14) nothing is added
    if precision == "fp64":
        assert np.allclose(h, want, rtol=1e-12, atol=2e-14 * max(q.size, 1))
    hc, tc, nc = m.chain()   # FP64 sums of the same weights in another order
    assert np.allclose(h, hc, rtol=1e-12, atol=0.0)
    assert count == nc
    assert np.isclose(total, tc, rtol=1e-12, atol=0.0)
    assert np.isclose(total, q.sum(), rtol=1e-12, atol=0.0)
