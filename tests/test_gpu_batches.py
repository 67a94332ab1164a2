"""A tilt series gives the same images and exit waves, bit for bit, whether its
orientations run in one batch or a few at a time, where the transmit reads whole
rows of the transmissions (nmode 1 and 2, a spherical incident wave): exit waves
and rotated image planes of the batch before pass through the same buffers and
leave their out-of-band columns filled."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,what", [
    (256, 256, "nmode 1"), (512, 512, "nmode 1"), (256, 512, "nmode 2"), (64, 64, "nmode 2"),
    (512, 512, "exit waves"), (256, 512, "exit waves"), (512, 256, "rotated planes"),
    (256, 256, "rotated planes")])
def test_batches_equal(ctx, msk, nx, ny, what):
    rng = np.random.default_rng(nx + ny)
    n, na = 80, 12
    x, y = rng.uniform(7.0, 25.0, (2, n)).astype(np.float32)
    z = rng.uniform(0.2, 31.0, n).astype(np.float32)
    at = (rng.choice([6, 7, 8, 16], n).astype(np.int32), x, y, z, np.ones(n, np.float32))
    rot = np.array([0.3])
    res = []
    for batch in (0, 5):
        s = msk.Series()
        s.nx, s.ny, s.ctblength, s.ctblengthz, s.v0, s.deltaz = nx, ny, 32.0, 32.0, 300.0, 4.0
        s.max_batch = batch
        if what[:5] == "nmode":
            s.nmode = int(what[-1])
        else:
            s.R1 = 50.0
        if what == "rotated planes":
            s.rotation = rot.ctypes.data
        defocus = [] if what == "exit waves" else [20.0]
        res.append(ctx.tilt_series(s, *at, np.linspace(0.0, 0.1, na), np.linspace(0.0, 0.1, na), defocus,
                                   want_exit=True))
    for one, few in zip(*res):
        assert np.array_equal(one.view(np.uint32), few.view(np.uint32))
        if one.dtype == np.float32 and one.size:
            assert np.abs(one).max() > 0
