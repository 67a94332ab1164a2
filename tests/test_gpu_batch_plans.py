"""A specimen batch settles the schedules of the passes it runs: the Debye-Waller pass's
where a specimen is damped only.  A schedule is kept for the life of a process, so the
batches run in one of their own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, %r)
import utr_public_gb300 as msk
from utr_public_gb300 import specimen as sp
ctx = msk.Context(0)
spec = sp.random_specimen(60, 30.0, 6.0, 24.0, 3)
s = msk.Series()
s.v0, s.deltaz = 200.0, 3.0
ang = np.array([0.0, 0.3])
for damped in (0, 1):
    s.lwobble, s.temperature = damped, 300.0
    if damped:
        spec.wobble = np.full(60, 0.07, np.float32)
    ctx.tilt_series_batch(s, [(spec, 128, ang, ang)], [20.0])
    plans = [msk.column_plan(0, 128, 128, p) for p in msk.COLUMN_PASSES]
    assert [p is not None for p in plans] == [True, True, True, bool(damped)], plans
""" % ROOT


def test_only_the_passes_that_run():
    r = subprocess.run([sys.executable, "-c", SCRIPT], timeout=300, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
