"""The per-kernel profile of a small call names its passes for what they are: the wave
chain of a group of slices, the row pass that makes its transmissions, and exit-wave work
only where exit waves are asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 512])
@pytest.mark.parametrize("want_exit", [False, True])
def test_small_call(ctx, msk, n, want_exit):
    rng = np.random.default_rng(n)
    at = (rng.choice([6, 8], 40).astype(np.int32), *rng.uniform(8.0, 32.0, (3, 40)).astype(np.float32),
          np.ones(40, np.float32))
    s = msk.Series()
    s.nx = s.ny = n
    s.ctblength = s.ctblengthz = 40.0
    s.v0, s.deltaz = 200.0, 4.0
    run = lambda: ctx.tilt_series(s, *at, [0.2], [0.1], [20.0], want_exit=want_exit)
    run()  # schedules chosen (where they are 16-point ones, 512^2 runs in a launch per pass)
    plans = msk.row_plan(0, n, n), msk.column_plan(0, n, n, "propagate")
    ctx.profile(True)
    try:
        run()
        kinds = ctx.profile_read()
    finally:
        ctx.profile(False)
    chain = n == 128 or all(p["points_per_thread"] == 32 for p in plans)
    assert ("wave_chain" in kinds) == ("row_band_inverse" in kinds) == chain
    assert ("row_exit" in kinds) == want_exit
    if chain:
        # (a group of slices without atoms has a wave chain alone)
        assert kinds["wave_chain"][0] >= kinds["row_band_inverse"][0] == kinds["row_splat"][0] > 0
        assert "col_propagate" not in kinds and "row_transmit" not in kinds
