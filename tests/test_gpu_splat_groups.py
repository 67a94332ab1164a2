"""The splat reads back only the pixel groups that atom windows reach and writes
rows without atoms from registers: atoms at the box edges (windows that wrap
around a row), windows as long as the row and longer, one atom alone, atoms of
occupancy zero, and grids whose band is narrower than the rows' own.  Exit
waves against the FP64 oracle within 1e-5."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

GRIDS = [(16, 16, 8.0), (32, 64, 6.5), (64, 64, 5.0), (128, 128, 40.0), (256, 1024, 33.0),
         (1024, 256, 33.0), (1024, 1024, 160.0), (1024, 1024, 21.0), (2048, 512, 90.0),
         (512, 2048, 90.0), (64, 4096, 60.0)]


@pytest.mark.parametrize("nx,ny,fov", GRIDS)
@pytest.mark.parametrize("kind", ["edges", "one", "empty_occ"])
def test_exit_wave(ctx, msk, oracle, nx, ny, fov, kind):
    rng = np.random.default_rng(nx + 3 * ny)
    f = np.float32(fov)
    edge = np.array([0.0, 0.01, 0.5, 0.99, 1.0])
    if kind == "one":
        xyz = np.array([[0.31], [0.002], [0.4]])
    else:
        xyz = np.stack([rng.choice(edge, 12), rng.choice(edge, 12), rng.uniform(0.1, 0.9, 12)])
    x, y, z = (np.minimum((q * fov).astype(np.float32), f) for q in xyz)
    z = (z * np.float32(6.0 / fov)).astype(np.float32)
    n = len(x)
    num = rng.choice([6, 8, 16], n).astype(np.int32)
    occ = np.ones(n, np.float32)
    if kind == "empty_occ":
        occ[::2] = 0.0
    s = msk.Series()
    s.nx, s.ny, s.ctblength, s.ctblengthz = nx, ny, fov, 6.0
    s.v0, s.deltaz = 300.0, 2.0
    _, ew, _ = ctx.tilt_series(s, num, x, y, z, occ, [0.0], [0.0], [10.0], want_exit=True)
    from oracle.oracle import SeriesParams
    p = SeriesParams()
    p.ax, p.ctblengthz, p.nx, p.ny, p.v0, p.deltaz = fov, 6.0, nx, ny, 300.0, 2.0
    p.aobj, p.max_slices, p.min_slice = 0.0, -1, 0
    _, ref, _ = oracle.orientation(p, num, x, y, z, occ, 0.0, 0.0, np.array([10.0]), fp64=True,
                                   want_exit=True)
    assert rel_l2(ew[0, 0], ref) < 1e-5
