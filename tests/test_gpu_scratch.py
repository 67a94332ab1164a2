"""Device scratch of a call follows the call's own size, not that of the largest call
before it: a small Debye-Waller series after a large plain one needs its tables, a
schedule tuner's grids (64 of 128^2: 8 MiB) and its own spectra, not another copy of the
large call's transmissions (512 MiB a buffer)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["tilt_series", "calculate"])
def test_small_call_after_large(msk, how):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    n = 50
    xyz = rng.uniform(8.0, 32.0, (3, n)).astype(np.float32)
    at = (rng.choice([6, 7, 8], n).astype(np.int32), *xyz, np.ones(n, np.float32))
    wob = np.full(n, 0.07, np.float32)

    def series(g, na, dw):
        s = msk.Series()
        s.nx = s.ny = g
        s.ctblength = s.ctblengthz = 40.0
        s.v0, s.deltaz = 200.0, 10.0
        if dw:
            s.lwobble, s.temperature, s.wobble = 1, 300.0, wob.ctypes.data
        im = torch.empty((na, 1, g, g), device="cuda")
        c.tilt_series(s, *at, np.linspace(0.0, 0.1, na), np.zeros(na), [0.0], images=im)
        return im

    def small():
        if how == "tilt_series":
            return series(128, 2, True).cpu().numpy()
        par = msk.make_param(40.0, 40.0, 128, 128, 200.0, 10.0)
        return c.calculate(par, *at, 40.0, 40.0, wobble=wob, lwobble=1)

    c = msk.Context(0)
    want = small()
    c.close()
    c = msk.Context(0)
    try:
        series(1024, 64, False)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        got = small()
        assert free - torch.cuda.mem_get_info()[0] < 64 << 20
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    finally:
        c.close()
