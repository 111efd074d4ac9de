"""A resident PCG whose blocks do not all start in time (FLOF_OPT_RESIDENT_POLLS
0: none waits) leaves the level to the chained kernels, from where it stood."""
import numpy as np
import pytest

from test_gpu_cg_step import cg64

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    import ofblend_gb300 as F
    from ofblend_gb300 import _lib

    c = F.Context(0)
    c.set_option(_lib.FLOF_OPT_RESIDENT_POLLS, 0)
    return c


def pair(dims):
    rng = np.random.default_rng(sum(dims))
    X, Y, Z, T = dims
    base = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
    for ax in range(4):  # a smooth field of the solver's input magnitude
        base = (base + np.roll(base, 1, ax)).astype(np.float32) * np.float32(0.5)
    i0 = base * np.float32(0.02)
    return i0, np.roll(i0, 1, axis=3) + np.float32(0.001)


# one block and several; each launch shape (cells per SM up to 256, 1024, 6144, more)
@pytest.mark.parametrize("dims", [(3, 3, 3, 3), (5, 4, 3, 6), (21, 17, 16, 9), (56, 55, 40, 3), (80, 83, 85, 3),
                                  (110, 108, 113, 3)])
def test_left_level_is_solved_by_the_chain(ctx, dims):
    import ofblend_gb300 as F

    i0, i1 = pair(dims)
    g0 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i0)
    g1 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i1)
    n = 5
    v = F.Grid4Vec4(dims=dims, ctx=ctx)
    ctx.profile(True)
    it, _ = F.opticalFlow4d(v, g0, g1, wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-12, cgMaxIter=n)
    names = {r[0] for r in ctx.profile_records()}
    ctx.profile(False)
    assert {"cg_resident", "cg_matvec", "cg_step"} <= names
    want = cg64(i0, i1, 0.001, 0.0001, it)
    got = v.to_numpy().astype(np.float64)
    # as for the chained kernels alone: 3 x 20 roundings an iteration
    assert it <= n and np.linalg.norm(got - want) <= 60 * n * 2.0 ** -24 * np.linalg.norm(want)


@pytest.mark.parametrize("kw", [dict(), dict(precision="mixed"), dict(solver="mg")])
def test_solves_agree_with_the_resident_ones(ctx, kw):
    """Every caller of the resident PCG: the plain solve, both starts of the
    mixed one (its corrections are solved from zero), and the finish of the
    multigrid solve (from the x that it stands at)."""
    import ofblend_gb300 as F

    dims = (24, 22, 20, 16)
    i0, i1 = pair(dims)
    out = []
    for c in (F.Context(0), ctx):
        if kw.get("solver") == "mg":
            c.set_mg_params(max_iter=2)  # stops short: the plain PCG finishes
        g0, g1 = F.Grid4Real(dims=dims, ctx=c).from_numpy(i0), F.Grid4Real(dims=dims, ctx=c).from_numpy(i1)
        v = F.Grid4Vec4(dims=dims, ctx=c)
        F.opticalFlowMultiscale4d(v, g0, g1, wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-5, postVelBlur=4, cfl=999,
                                  multiStep=3, minGridSize=10, resetBndWidth=0.1, **kw)
        assert c.mg_fallbacks() > 0 or "solver" not in kw
        out.append(v.to_numpy().astype(np.float64))
    # the deformation tolerance of the package
    assert np.linalg.norm(out[1] - out[0]) <= 1e-4 * np.linalg.norm(out[0])


def test_batch_workers_take_the_option(ctx):
    import ofblend_gb300 as F

    dims = (16, 14, 12, 10)
    i0, i1 = pair(dims)
    g0, g1 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i0), F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i1)
    vs = [F.Grid4Vec4(dims=dims, ctx=ctx) for _ in range(5)]
    kw = dict(wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-3, minGridSize=8)
    F.opticalFlowMultiscale4d_batch(vs[1:], [g0] * 4, [g1] * 4, workers=3, **kw)
    F.opticalFlowMultiscale4d(vs[0], g0, g1, **kw)
    for v in vs[1:]:
        assert np.array_equal(v.to_numpy(), vs[0].to_numpy())
