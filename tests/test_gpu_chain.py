"""The wave chain of small calls in one launch per slice group: clusters for grids of
64^2 to 256^2 (more CTAs than SMs, too), one cooperative launch for a lone unit of
512^2 or 1024^2.
MSK_SMALL_GRID=0 selects the launch-per-pass loop, whose 32-point plans the wide
kernel shares (the same bits); the cluster kernel's plan is another (relative L2
2e-6), and both are within 1e-5 of the FP64 oracle.  An incident wave of white noise
fills the band: the FP32 roundings of the two propagator tables and of the twiddles
are the same in every slice and add up coherently, at most u = 2^-24 a table entry,
so 2 u a slice against FP64 and u a slice between two plans.  Enough slices for several
groups, slices without atoms at both ends and in the middle, a plane and an
arbitrary incident wave, the Debye-Waller branch, odd unit counts, a thin last
slice."""
import os

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def both(fn):
    one = fn()
    os.environ["MSK_SMALL_GRID"] = "0"
    try:
        return one, fn()
    finally:
        os.environ.pop("MSK_SMALL_GRID", None)


def same(n, a, b, slack=0.0):
    if n > 256:
        return np.array_equal(a.view(np.uint32), b.view(np.uint32))
    return rel_l2(a, b) < 2e-6 + slack


def atoms_with_gaps(n):
    rng = np.random.default_rng(n)
    z = np.concatenate([rng.uniform(3.1, 8.0, 40), rng.uniform(12.7, 17.4, 40)])
    xy = rng.uniform(6.0, 34.0, (2, 80))
    return (rng.choice([6, 7, 8, 16], 80).astype(np.int32), *xy.astype(np.float32), z.astype(np.float32),
            np.ones(80, np.float32))


@pytest.mark.parametrize("wave", [False, True])
@pytest.mark.parametrize("n,dz", [(64, 0.7), (128, 0.3), (256, 0.06), (512, 0.19), (1024, 0.9)])
def test_calculate(ctx, msk, oracle, n, dz, wave):
    at = atoms_with_gaps(n)
    param = msk.make_param(40.0, 40.0, n, n, 200.0, dz)
    kw, slack = {}, 0.0
    if wave:
        slack = 2.0**-24 * 22.0 / dz
        ph = np.random.default_rng(3).uniform(0, 2 * np.pi, (n, n))
        kw["wave0"] = np.stack([np.cos(ph), np.sin(ph)], -1).astype(np.float32)
    got, loop = both(lambda: ctx.calculate(param, *at, 40.0, 22.0, **kw))
    assert same(n, got, loop, slack)
    if wave:
        kw["wave0"] = kw["wave0"].astype(np.float64)
    ref = oracle.calculate(param, *at, 40.0, 22.0, fp64=True, **kw)
    assert rel_l2(got, ref) < 1e-5 + 2 * slack


@pytest.mark.parametrize("dw", [False, True])
@pytest.mark.parametrize("n,na", [(64, 1), (64, 7), (64, 200), (128, 3), (128, 19), (256, 5), (512, 1),
                                  (1024, 1)])
def test_tilt_series(ctx, msk, n, na, dw):
    at = atoms_with_gaps(n)
    s = msk.Series()
    s.nx = s.ny = n
    s.ctblength, s.ctblengthz, s.v0, s.deltaz = 40.0, 22.0, 200.0, 0.8
    wob = np.full(80, 0.07, np.float32)
    if dw:
        s.lwobble, s.temperature, s.wobble = 1, 300.0, wob.ctypes.data
    run = lambda: ctx.tilt_series(s, *at, np.linspace(0.0, 2.0, na), np.linspace(0.1, 0.4, na), [0.0, 30.0],
                                  want_exit=True)
    (img, ew, kept), (img0, ew0, kept0) = both(run)
    assert np.array_equal(kept, kept0)
    for a in range(na):
        assert same(n, ew[a], ew0[a]) and same(n, img[a], img0[a]), a
