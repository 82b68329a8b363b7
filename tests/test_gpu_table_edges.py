"""GPU table fill at the sizes where its layout changes: rows shorter than a
warp, at and beyond the widest that passes through shared memory (1024
intervals; wider rows evaluate their values twice), one row, and row counts
around the block shapes; rows that are masked in part or whole."""
import numpy as np
import pytest

import mcd_oracle as O
from mcd import _lib, tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nW", [2, 3, 32, 33, 34, 97, 1024, 1025, 1026, 1500])
@pytest.mark.parametrize("nE", [1, 7, 160])
@pytest.mark.parametrize("kind,sp", [("Moller", "Si"), ("Gryz", "Al"), ("Gryz", "Au")])
def test_fill_edges(kind, sp, nE, nW):
    m = _lib.material(sp)
    wmin = 100.0 if kind == "Moller" else float(m.shell_E[m.n_shells - 1])
    # the lowest energies leave no unmasked interval at all
    Es = np.linspace(1.5 * wmin, 20000.0, num=nE, dtype=np.float32)
    Ws = np.geomspace(wmin, (20000.0 - m.fermi_e) / 2, num=nW, dtype=np.float32)
    dt = tables.DeviceTable(kind, m, Ws, Es, "cuda", keep_fp64=True)
    cdf32, cdf64 = dt.cdf.cpu().numpy(), dt.cdf64.cpu().numpy()
    ocdf, valid = O.table_cdf(kind, O.Material(sp), Ws, Es)
    assert np.array_equal(dt.nvalid.cpu().numpy(), valid.sum(axis=1))
    assert np.all(cdf64[~valid] == 0) and np.all(cdf32[~valid] == 0)
    if valid.any():
        # the oracle's sequential sums round within nW 2^-53; the fill's terms
        # are within a few rounding errors each
        assert np.max(np.abs(cdf64[valid] - ocdf[valid])) < 1e-13
    assert np.array_equal(cdf32, cdf64.astype(np.float32))
    # the guide: first unmasked entry at or above k/256
    g = dt.guide.cpu().numpy().view(np.uint16)
    q = np.arange(_lib.GUIDE + 1, dtype=np.float32) / np.float32(_lib.GUIDE)
    for r in range(nE):
        nv = int(valid[r].sum())
        assert np.array_equal(g[r], np.searchsorted(cdf32[r, :nv], q))
