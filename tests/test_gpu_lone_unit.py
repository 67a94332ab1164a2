"""A unit of 512^2 or 1024^2 gives the same bits alone (where its wave chain may run in one
launch) as among several (where it runs in a launch per pass), whatever schedules the
column and row passes have: chosen by timing, or fixed by MSK_COL_TILE or MSK_ROW_PLAN.
A schedule is kept for the life of a process, so each runs in its own."""
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
ctx = msk.Context(0)
for n in (512, 1024):
    rng = np.random.default_rng(n)
    xyz = rng.uniform(8.0, 32.0, (3, 90)).astype(np.float32)
    at = (rng.choice([6, 7, 8, 16], 90).astype(np.int32), *xyz, np.ones(90, np.float32))
    s = msk.Series()
    s.nx = s.ny = n
    s.ctblength = s.ctblengthz = 40.0
    s.v0, s.deltaz = 200.0, 2.0
    angles = np.array([0.0, 0.4, 0.9])
    img, ew, _ = ctx.tilt_series(s, *at, angles, 0.5 * angles, [20.0], want_exit=True)
    for a in (0, 2):
        img1, ew1, _ = ctx.tilt_series(s, *at, angles[a:a + 1], 0.5 * angles[a:a + 1], [20.0], want_exit=True)
        assert np.array_equal(img1[0].view(np.uint32), img[a].view(np.uint32)), (n, a)
        assert np.array_equal(ew1[0].view(np.uint32), ew[a].view(np.uint32)), (n, a)
""" % ROOT


@pytest.mark.parametrize("var,value", [(None, None), ("MSK_ROW_PLAN", "1"), ("MSK_ROW_PLAN", "2"),
                                       ("MSK_COL_TILE", "1"), ("MSK_COL_TILE", "2"), ("MSK_COL_TILE", "3")])
def test_alone_as_among_several(var, value):
    env = {k: v for k, v in os.environ.items() if k not in ("MSK_ROW_PLAN", "MSK_COL_TILE")}
    if var:
        env[var] = value
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, timeout=300, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
