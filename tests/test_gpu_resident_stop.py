"""The resident PCG's iterates and the iteration it stops at, at every launch
shape: after a fixed number of iterations its x is that of the same iterations
in 64 bits, and a solve stops at the first iterate that meets the threshold."""
import numpy as np
import pytest

from test_gpu_cg_step import cg64
from test_gpu_resident import SIZES

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[d for d in SIZES if d != (131, 131, 131, 3)], ids=lambda d: "x".join(map(str, d)))
def solve(request):
    import ofblend_gb300 as F

    dims = request.param
    rng = np.random.default_rng(sum(dims))
    X, Y, Z, T = dims
    base = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
    for ax in range(4):  # a smooth field of the solver's input magnitude
        base = (base + np.roll(base, 1, ax)).astype(np.float32) * np.float32(0.5)
    i0 = base * np.float32(0.02)
    i1 = np.roll(i0, 1, axis=3) + np.float32(0.001)
    g0, g1 = F.Grid4Real(dims=dims).from_numpy(i0), F.Grid4Real(dims=dims).from_numpy(i1)
    v = F.Grid4Vec4(dims=dims)

    def run(accuracy, cap):
        v.clear()
        it, res = F.opticalFlow4d(v, g0, g1, wSmooth=0.001, wEnergy=0.0001, cgAccuracy=accuracy, cgMaxIter=cap)
        return it, res, v.to_numpy().astype(np.float64)

    run.fields = i0, i1
    return run


def test_iterates_match_64_bits(solve):
    for n in (1, 2, 5):
        it, _, got = solve(1e-12, n)
        # one cell ends by itself: its system has four unknowns
        assert it == n or got.size == 4 * 81
        want = cg64(*solve.fields, 0.001, 0.0001, it)
        # q, r, p and x are each rounded at some 20 places an iteration, and an
        # iteration carries the errors of those before it
        assert np.linalg.norm(got - want) <= 60 * it * 2.0 ** -24 * np.linalg.norm(want)


def test_stops_at_the_first_iterate_below_the_threshold(solve):
    for accuracy in (0.3, 0.03):
        it, res, _ = solve(accuracy, 1000)
        assert 0 < it < 1000 and res <= accuracy
        if it > 1:
            before, left, _ = solve(accuracy, it - 1)
            assert before == it - 1 and left > accuracy
