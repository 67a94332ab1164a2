"""Reconstruction from orientations about y alone (gridding and Fourier rows in one
pass, rows of 256 to 1024 points, enough of them and a depth of half the width or
more; the others take the general path both times) against the general path: a rotation of 360
degrees about z for the first orientation leaves every coordinate as it is
(sin is 2e-16 there) but is not an orientation about y alone.

The two differ in the order of FP32 sums of at most a few hundred terms and in the
radix plan of one of three FFTs: 1e-6 relative L2 each at most (u sqrt(terms),
u log2 N), 3e-6 together; with the noise filter, whose arc tangent has a slope of
100, 2e-5.  Both Ewald options, an off-centre rotation axis, angles that put whole
pixel rows on one voxel row, negative and beyond half a turn, volumes shallower
than a CTA's rows or not square, a single image."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_utr import as_msk
from utr_cases import images, params

pytestmark = pytest.mark.gpu

ANGLES = {1: [0.0], 2: [90.0, 0.02], 31: np.linspace(0.0, 174.0, 31), 40: np.linspace(-200.0, 300.0, 40)}


@pytest.mark.parametrize("escc", [0, 1])
@pytest.mark.parametrize("nx,ny,nz,n,kw", [
    (64, 64, 64, 31, {}), (64, 32, 16, 40, {"nsr": 0.03}), (128, 64, 32, 40, {"dxc": 1.3, "dzc": -0.7}),
    (256, 16, 128, 31, {}), (512, 16, 512, 40, {"nsr": 0.02}), (512, 32, 16, 2, {}),
    (1024, 16, 256, 31, {"dyc": 0.4}), (256, 64, 256, 1, {}), (32, 32, 32, 31, {}), (2048, 16, 16, 2, {}),
    (256, 128, 128, 31, {}), (512, 512, 16, 2, {}), (256, 512, 16, 40, {}),
    (512, 64, 256, 40, {"dxc": 1.3, "dzc": -0.7}), (1024, 16, 512, 31, {"dyc": 0.4}),
    (256, 16, 1024, 40, {})])
def test_tilt_rows(ctx, msk, nx, ny, nz, n, kw, escc):
    p = params(nx, ny, nz, escc=escc, **kw)
    im = images(p, n, seed=nx + nz)
    ang = np.stack([np.zeros(n), ANGLES[n]], 1)
    one = ctx.utr_reconstruct(as_msk(msk, p), ang, np.full(n, 300.0), im)
    ang[0, 0] = 360.0
    ref = ctx.utr_reconstruct(as_msk(msk, p), ang, np.full(n, 300.0), im)
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0
    assert rel_l2(one, ref) < (2e-5 if "nsr" in kw else 3e-6)
