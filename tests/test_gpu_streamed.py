"""Streamed passes (one CTA per SM working through a launch's rows), which a
launch with enough rows takes, against the plain ones that a small call takes:
the same transforms with the same roundings, so every image is the same bit for
bit, and within 1e-5 of the FP64 oracle.  Grids: rows of 64 to 1024 points, the
band limited by the rows' own axis and by the other one (narrower segments),
numbers of rows that do not divide evenly among the warps, transmission only
(whole rows, no band) and the scattered form."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# nx, ny, orientations, nmode: above and (the last) just below the streaming rule
GRIDS = [(1024, 1024, 11, 0), (512, 1024, 19, 0), (1024, 512, 19, 0), (512, 512, 37, 1),
         (256, 256, 149, 0), (64, 256, 587, 0), (256, 64, 601, 0), (128, 128, 583, 0),
         (1024, 1024, 8, 0)]


def series(msk, nx, ny, nmode, fov):
    s = msk.Series()
    s.nx, s.ny = nx, ny
    s.ctblength, s.ctblengthz = fov, 8.0
    s.v0, s.deltaz, s.nmode = 300.0, 4.0, nmode
    return s


def atoms(fov, seed):
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(0.2 * fov, 0.8 * fov, size=(3, 60)).astype(np.float32)
    xyz[2] = rng.uniform(0.5, 7.5, 60)
    return (rng.choice([6, 7, 8, 16], 60).astype(np.int32), *xyz, np.ones(60, np.float32))


@pytest.mark.parametrize("nx,ny,na,nmode", GRIDS)
def test_streamed_equals_plain(ctx, msk, oracle, nx, ny, na, nmode):
    fov = 32.0
    at = atoms(fov, nx + ny)
    angz, angy = np.linspace(0.0, 3.0, na), np.zeros(na)
    run = lambda some: ctx.tilt_series(series(msk, nx, ny, nmode, fov), *at, angz[some],
                                       angy[some], [20.0])
    img, kept = run(slice(None))
    few = 5 if nx * ny >= 1 << 18 else 64  # calls too small for the streaming rule
    for some in (slice(0, few), slice(na - few, na)):
        img2, kept2 = run(some)
        assert np.array_equal(kept[some], kept2)
        assert np.array_equal(img[some].view(np.uint32), img2.view(np.uint32))
    if nmode:
        return
    from oracle.oracle import SeriesParams
    p = SeriesParams()
    p.ax, p.ctblengthz, p.nx, p.ny, p.v0, p.deltaz = fov, 8.0, nx, ny, 300.0, 4.0
    p.aobj, p.max_slices, p.min_slice = 0.0, -1, 0
    for a in (0, na - 1):
        ref, _, _ = oracle.orientation(p, *at, angz[a], angy[a], np.array([20.0]), fp64=True,
                                       want_exit=True)
        assert rel_l2(img[a, 0], ref[0]) < 1e-5, a


def test_streamed_scattered_form(ctx, msk):
    torch = pytest.importorskip("torch")
    g = torch.Generator().manual_seed(3)
    v = (torch.rand((21, 3, 512, 512), generator=g) * 40.0).cuda()
    v *= (torch.rand((21, 3, 512, 1), generator=g) < 0.7).cuda()
    imgs = []
    for batch in (0, 4):
        st = msk.Stack()
        st.nx = st.ny = 512
        st.ax = st.by = 40.0
        st.v0, st.deltaz, st.nslices, st.max_batch = 200.0, 1.0, 3, batch
        out = torch.empty((21, 1, 512, 512), device="cuda")
        ctx.stack_images(st, v, [30.0], images=out)
        imgs.append(out)
    assert torch.equal(imgs[0], imgs[1])
