"""The ring of search directions takes its buffers as the pool has them: what an
earlier call left there, border rows included, must not reach the solve."""
import numpy as np
import pytest

from test_gpu_cg_step import cg64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(134, 133, 132, 3), (43, 45, 41, 42), (37, 70, 33, 41)])
@pytest.mark.parametrize("n", [0, 1, 2, 4, 7])
def test_solve_ignores_what_the_pool_holds(dims, n):
    import ofblend_gb300 as F

    ctx = F.Context(0)
    X, Y, Z, T = dims
    rng = np.random.default_rng(n)
    base = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
    for ax in range(4):  # a smooth field of the solver's input magnitude
        base = (base + np.roll(base, 1, ax)).astype(np.float32) * np.float32(0.5)
    i0 = base * np.float32(0.02)
    i1 = np.roll(i0, 1, axis=3) + np.float32(0.001)
    g0, g1 = (F.Grid4Real(dims=dims, ctx=ctx).from_numpy(a) for a in (i0, i1))
    v = F.Grid4Vec4(dims=dims, ctx=ctx)
    kw = dict(wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-12, cgMaxIter=n)
    F.opticalFlow4d(v, g0, g1, **kw)
    first = v.to_numpy()
    # the same buffers again, full of NaN: a solve of a NaN field writes g, r, p,
    # q and the ring, a blur of one its scratch grids
    bad = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(np.full_like(i1, np.nan))
    w = F.Grid4Vec4(dims=dims, ctx=ctx).from_numpy(np.full(i1.shape + (4,), np.nan, np.float32))
    F.opticalFlow4d(w, g0, bad, **kw)
    for blur in (1, 2):
        w.from_numpy(np.full(i1.shape + (4,), np.nan, np.float32))
        F.gaussianBlur4d(w, 1.0, blur)
    v.clear()
    it, _ = F.opticalFlow4d(v, g0, g1, **kw)
    got = v.to_numpy()
    assert it == n and np.array_equal(got, first)
    if n:
        want = cg64(i0, i1, 0.001, 0.0001, n)
        assert np.linalg.norm(got - want) <= 60 * n * 2.0 ** -24 * np.linalg.norm(want)
