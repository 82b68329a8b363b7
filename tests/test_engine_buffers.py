"""What the host side makes of a run's device buffers (on CPU tensors)."""
import ctypes as C

import numpy as np
import pytest

from mcd import _lib, engine


def test_tally_bytes():
    t = _lib.Tally()
    t.outcome[1] = 7
    t.sum_E_bks = 2.5
    t.hist_T[3] = 9
    raw = bytes(t)
    for buf in (raw, raw + b"xyz", np.frombuffer(raw, dtype=np.uint8), bytearray(raw)):
        d = engine.tally_from_bytes(buf)
        assert d["bks"] == 7 and d["sum_E_bks"] == 2.5 and d["hist_T"][3] == 9
    for n in (0, 8, 240, C.sizeof(_lib.Tally) - 8, C.sizeof(_lib.Tally) - 1):
        with pytest.raises(ValueError):
            engine.tally_from_bytes(raw[:n])
