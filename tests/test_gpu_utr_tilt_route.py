"""Which orientations and volumes take the one pass of gridding and Fourier rows, told by
the profile (the general path launches a gridding kernel), and its result against the
general path (a rotation of 360 degrees about z for one orientation) at the angles
hardest for the search of a pixel row's run: along z, where every pixel has a voxel row of
its own, nearly flat, where a row lies in one or two, and a half turn.

The two differ in the order of FP32 sums and in the radix plan of one of three FFTs:
1e-6 relative L2 each at most (u sqrt(terms), u log2 N), 3e-6 together."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_utr import as_msk
from utr_cases import images, params

pytestmark = pytest.mark.gpu

ANGLES = [(90.0, 0.02), (0.0, 90.0, 0.02, 180.0), (-90.0, 270.0, 89.98, 1e-7), (0.0,)]


def run(ctx, msk, p, im, ang):
    """The volume and whether the general gridding ran."""
    ctx.profile(True)
    try:
        vol = ctx.utr_reconstruct(as_msk(msk, p), ang, np.full(len(ang), 300.0), im)
        return vol, "utr_grid" in ctx.profile_read()
    finally:
        ctx.profile(False)


@pytest.mark.parametrize("escc", [0, 1])
@pytest.mark.parametrize("ys", ANGLES)
@pytest.mark.parametrize("nx,ny,nz", [(512, 64, 256), (256, 128, 128), (256, 64, 256), (1024, 16, 512),
                                      (256, 16, 1024)])
def test_one_pass(ctx, msk, nx, ny, nz, ys, escc):
    p = params(nx, ny, nz, escc=escc)
    im = images(p, len(ys), seed=nx + nz)
    ang = np.stack([np.zeros(len(ys)), ys], 1)
    one, general = run(ctx, msk, p, im, ang)
    assert not general
    ang[0, 0] = 360.0
    ref, general = run(ctx, msk, p, im, ang)
    assert general
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0
    assert rel_l2(one, ref) < 3e-6


@pytest.mark.parametrize("nx,ny,nz", [(128, 128, 128), (2048, 16, 16), (512, 512, 128), (256, 16, 128)])
def test_general_path(ctx, msk, nx, ny, nz):
    """Rows of another length, flat volumes, too few rows for the GPU."""
    p = params(nx, ny, nz)
    _, general = run(ctx, msk, p, images(p, 1), np.array([[0.0, 30.0]]))
    assert general
