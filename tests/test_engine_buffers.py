"""What the host side makes of a run's buffers."""
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


def held_bytes(a):
    """The host memory that keeping the array keeps alive."""
    while isinstance(a, np.ndarray) and a.base is not None:
        a = a.base
    return a.nbytes if isinstance(a, np.ndarray) else a.untyped_storage().nbytes()


def collected(n):
    import torch
    bufs = engine.RunBuffers(n, _lib.FP32, True)
    planes = torch.arange(3 * n, dtype=torch.float32, device="cuda")
    bufs.el["dir"].copy_(planes)
    bufs.el["last_pos"].copy_(planes + 1)
    bufs.el["n_events"].copy_(torch.arange(n, device="cuda"))
    return bufs, engine.collect(bufs).electrons


@pytest.mark.gpu
@pytest.mark.parametrize("n", [0, 1, 1000, 8191, 8192, 100003, 2 ** 18 - 1, 2 ** 18])
def test_rows_hold_no_more_than_they_need(n):
    bufs, rows = collected(n)
    want = np.arange(3 * n, dtype=np.float32).reshape(3, n).T
    assert np.array_equal(rows["dir"], want) and np.array_equal(rows["last_pos"], want + 1)
    assert np.array_equal(rows["n_events"], np.arange(n))
    assert list(rows) == ["outcome", "flags", "final_E", "dir", "last_pos", "max_z", "n_events"]
    # the columns of the middle sizes share a buffer that holds nothing larger
    columns = sum(a.nbytes for k, a in rows.items() if k not in ("dir", "last_pos")) + C.sizeof(_lib.Tally) + 8 * 512
    for k, a in rows.items():
        own = k in ("dir", "last_pos") or not 8192 <= n < 2 ** 18
        assert a.flags.writeable and a.flags.c_contiguous, k
        assert held_bytes(a) == a.nbytes if own else held_bytes(a) <= columns, k


@pytest.mark.gpu
@pytest.mark.parametrize("n", [50000, 300000])
def test_large_rows_cross_the_link_once(monkeypatch, n):
    import torch
    crossed = []
    cpu = torch.Tensor.cpu

    def counted(t, *a, **k):
        crossed.append(t.numel() * t.element_size())
        return cpu(t, *a, **k)

    bufs, _ = collected(n)
    monkeypatch.setattr(torch.Tensor, "cpu", counted)
    rows = engine.collect(bufs).electrons
    # the tally, status and cursor and five columns, each rounded up to 512
    assert sum(crossed) <= sum(a.nbytes for a in rows.values()) + C.sizeof(_lib.Tally) + 8 * 512
