"""The host sort by z gives the reference's Shell-sort permutation, ties included: a
radix sort with counting walks, or the insertion passes for few atoms, few planes
or NaN.  Every array moves as the oracle's literal loops move it; sizes at the
edges of the rule (128) and of the gap sequence."""
import numpy as np
import pytest


def kinds(rng, n):
    u = rng.uniform(-5.0, 160.0, n).astype(np.float32)
    zero = u.copy()
    zero[rng.random(n) < 0.05] = 0.0
    zero[rng.random(n) < 0.05] = -0.0
    bad = u.copy()
    bad[rng.random(n) < 0.02] = np.nan
    far = u.copy()
    far[rng.random(n) < 0.04] = np.inf
    far[rng.random(n) < 0.04] = -np.inf
    return {"random": u, "rounded": np.round(u, 2), "planes": np.floor(u / 16), "rows": np.floor(u),
            "zeros": zero, "nan": bad, "inf": far, "falling": -np.arange(n, dtype=np.float32)}


@pytest.mark.parametrize("n", [0, 1, 2, 9, 10, 127, 128, 129, 361, 1093, 3000, 20000])
def test_sort_order(msk, oracle, n):
    rng = np.random.default_rng(n)
    x, y, occ = (rng.uniform(0.0, 9.0, n).astype(np.float32) for _ in range(3))
    Z = rng.integers(1, 104, n).astype(np.int32)
    for kind, z in kinds(rng, n).items():
        got, ref = (lib.sort_by_z(Z, x, y, z, occ) for lib in (msk, oracle))
        for a, b in zip(got, ref):
            assert np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32)), kind
