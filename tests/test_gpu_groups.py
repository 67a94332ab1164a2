"""Slice groups: with few units in a call the transmissions of several slices are
made in one launch per pass (the plain, phonon and Debye-Waller branches).  A
call's images and exit waves are the same bit for bit whether its units run
together (few slices a group, or none) or a few at a time (many slices a group),
and within 1e-5 of the FP64 oracle.  Slices without atoms at both ends of the box
and in the middle, orientation counts that leave ragged groups, a grid that is
not square."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def make(msk, nx, ny, kind, natom):
    s = msk.Series()
    s.nx, s.ny, s.ctblength, s.ctblengthz = nx, ny, 40.0, 22.0
    s.v0, s.deltaz = 200.0, 1.0
    wob = np.full(natom, 0.07, np.float32)
    if kind == "dw":
        s.lwobble, s.temperature, s.wobble = 1, 300.0, wob.ctypes.data
    return s, wob


@pytest.mark.parametrize("kind", ["plain", "dw", "phonon"])
@pytest.mark.parametrize("nx,ny,na", [(512, 512, 7), (256, 1024, 5), (1024, 64, 11), (32, 32, 33)])
def test_groups(ctx, msk, oracle, nx, ny, na, kind):
    rng = np.random.default_rng(nx + ny)
    n = 90
    x, y = (rng.uniform(8.0, 32.0, n).astype(np.float32) for _ in range(2))
    z = np.concatenate([rng.uniform(3.1, 9.0, n // 2), rng.uniform(13.2, 18.0, n - n // 2)]).astype(np.float32)
    num = rng.choice([6, 7, 8, 16], n).astype(np.int32)
    occ = np.ones(n, np.float32)
    s, wob = make(msk, nx, ny, kind, n)
    nc = 3 if kind == "phonon" else 1
    disp = rng.normal(0, 0.05, (nc, 3, n)).astype(np.float32) if kind == "phonon" else None
    angz = np.linspace(0.0, 2.0, na)
    run = lambda some: ctx.tilt_series(s, num, x, y, z, occ, angz[some], np.zeros(len(angz[some])),
                                       [15.0], nconfig=nc, displacements=disp, want_exit=True)
    img, ew, kept = run(slice(None))
    for a in (0, na - 1):
        img1, ew1, _ = run(slice(a, a + 1))
        assert np.array_equal(img1[0].view(np.uint32), img[a].view(np.uint32))
        assert np.array_equal(ew1[0].view(np.uint32), ew[a].view(np.uint32))
    if kind != "plain":
        return
    from oracle.oracle import SeriesParams
    p = SeriesParams()
    p.ax, p.ctblengthz, p.nx, p.ny, p.v0, p.deltaz = 40.0, 22.0, nx, ny, 200.0, 1.0
    p.aobj, p.max_slices, p.min_slice = 0.0, -1, 0
    _, ref, _ = oracle.orientation(p, num, x, y, z, occ, angz[-1], 0.0, np.array([15.0]), fp64=True,
                                   want_exit=True)
    assert rel_l2(ew[-1, 0], ref) < 1e-5


def test_one_unit_calculate(ctx, msk, oracle):
    """calculate() on a grid beyond the cluster kernel's: an arbitrary incident wave, whose
    first transmit reads whole rows, and the Debye-Waller branch."""
    rng = np.random.default_rng(4)
    n = 60
    xyz = rng.uniform(5.0, 25.0, (3, n)).astype(np.float32)
    at = (rng.choice([6, 8], n).astype(np.int32), *xyz, np.ones(n, np.float32))
    param = msk.make_param(30.0, 30.0, 512, 512, 200.0, 1.0)
    ph = rng.uniform(0, 2 * np.pi, (512, 512))
    w0 = np.stack([np.cos(ph), np.sin(ph)], -1).astype(np.float32)
    for wave in (None, w0):
        got = ctx.calculate(param, *at, 30.0, 30.0, wave0=wave)
        ref = oracle.calculate(param, *at, 30.0, 30.0, fp64=True,
                               **({} if wave is None else {"wave0": wave.astype(np.float64)}))
        assert rel_l2(got, ref) < 1e-5
