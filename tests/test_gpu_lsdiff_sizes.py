"""calcLsDiff4d over box sizes around its launch shape (four cells per thread
and trip): fewer cells than a block, remainders of a trip, several trips, and
calls in sequence (each answer is its own call's), against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bnd", [0, 1])
def test_calc_ls_diff_sizes(gpu, orc, bnd):
    import ofblend_gb300 as F
    rng = np.random.default_rng(5)
    for dims in [(3, 3, 3, 3), (5, 4, 3, 4), (16, 4, 4, 4), (17, 5, 4, 3), (33, 31, 9, 5), (40, 37, 33, 41)]:
        X, Y, Z, T = dims
        a = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
        b = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
        out = F.Grid4Real(dims=dims)
        got = F.calcLsDiff4d(F.Grid4Real(dims=dims).from_numpy(a), F.Grid4Real(dims=dims).from_numpy(b), out=out,
                             correction=0.7, bnd=bnd)
        s = (slice(bnd, -bnd if bnd else None),) * 4
        same = ((a < 0) & (b < 0)) | ((a >= 0) & (b >= 0))
        d = np.where(same, np.float32(0), np.minimum(np.abs(a - b) * np.float32(0.7), np.float32(1)))
        want = np.float32(d[s].astype(np.float64).sum() * 1e6 / d[s].size)
        # the sum is in double; another order of it moves the float by one ulp at most
        assert abs(got - want) <= np.spacing(want)
        full = np.zeros_like(a)
        full[s] = d[s]
        assert np.array_equal(out.to_numpy(), full)
