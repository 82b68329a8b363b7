"""Batches whose constants and drain seats just fit the shared memory a block
has without asking for more: the run-down kernel's own static arrays count too.
Each size runs in a process of its own, where no larger batch has raised the
limit before, and is compared with the launch that has no run-down kernel."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SCRIPT = """
import sys
sys.path[:0] = [{here!r}, {pkg!r}, {oracle!r}]
import test_zz_no_alloc as T
from mcd import _lib, engine
from _gpu_util import input_par
n, tune = {n}, _lib.Tune(256, 0, 1, 2, 0)
sims = [dict(input_par(("Al", "Si")[k % 2], 5000.0, 1000.0, 0.0), num_el=40 + k) for k in range(n)]
b = engine.Batch(sims, seed=3)
got, st = b.run(tune)
assert [sum(t[o] for o in ("bks", "abs", "trsm", "long")) for t in got] == [s["num_el"] for s in sims]
ref, st_ref = T._noalloc(b, tune)
T._same(got, ref)
assert st == st_ref
"""


@pytest.mark.parametrize("n", [42, 43, 44, 45])
def test_batch_at_the_shared_memory_line(n):
    root = os.path.dirname(HERE)
    code = SCRIPT.format(here=HERE, pkg=os.path.join(root, "mc-discrete_gb300"), oracle=os.path.join(root, "oracle"), n=n)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
