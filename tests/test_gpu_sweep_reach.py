"""The projection's sweeps leave out tiles that no marked cell can reach yet:
the whole correction against the plain-load sweeps (which visit every cell),
bit for bit, on grids of several tiles along each axis whose marked cells are a
thin layer, a far corner, or none at all, with few and many sweeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kind, dims, vmax):
    X, Y, Z, T = dims
    y = np.arange(Y, dtype=np.float32)[None, None, :, None]
    x = np.arange(X, dtype=np.float32)[None, None, None, :]
    shape = (T, Z, Y, X)
    if kind == "layer":
        i0 = np.broadcast_to(np.clip(y - 7.3, -4, 4), shape)
        i1 = np.broadcast_to(np.clip(y - 8.1, -4, 4), shape)
    elif kind == "corner":
        i0 = np.broadcast_to(np.clip(np.hypot(x - X + 5, y - Y + 5) - 3, -4, 4), shape)
        i1 = np.broadcast_to(np.clip(np.hypot(x - X + 6, y - Y + 5) - 3, -4, 4), shape)
    else:
        i0 = np.full(shape, 4.0, np.float32)
        i1 = np.full(shape, -4.0, np.float32)
    rng = np.random.default_rng(X)
    v = (rng.standard_normal(shape + (4,)) * 0.1).astype(np.float32)
    v[T // 2, Z // 2, Y // 2, X // 2, 0] = vmax  # sets the sweep count, int(max |v| + 4)
    return i0.astype(np.float32) * np.float32(0.2), i1.astype(np.float32) * np.float32(0.2), v


@pytest.mark.parametrize("kind", ["layer", "corner", "none"])
@pytest.mark.parametrize("dims,vmax", [((40, 70, 9, 19), 2.0), ((70, 37, 11, 12), 30.0), ((17, 90, 6, 33), 9.0)])
@pytest.mark.parametrize("solver", ["direct", "separable"])
def test_sweeps_match_plain_loads(kind, dims, vmax, solver):
    import ofblend_gb300 as F
    from ofblend_gb300 import _lib
    ctx = F.Context(0)
    i0, i1, v0 = _case(kind, dims, vmax)
    g0 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i0)
    g1 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i1)
    got = []
    for tma in (0, 1):
        ctx.set_option(_lib.FLOF_OPT_SLAB_TMA, tma)
        v = F.Grid4Vec4(dims=dims, ctx=ctx).from_numpy(v0)
        d = F.Grid4Vec4(dims=dims, ctx=ctx)
        if solver == "direct":
            F.corrVelsOf4d(d, v, g0, None, g1, threshPhi=4.0, postVelBlur=4.0, resetBndWidth=0.05, maxIter=40)
        else:  # the separable sweeps are reached through the solve's final projection
            F.opticalFlowMultiscale4d(v, g0, g1, wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-2, postVelBlur=2,
                                      minGridSize=200, multiStep=1, blurType=2, doFinalProject=True,
                                      resetBndWidth=0.05)
        got.append((v.to_numpy(), d.to_numpy()))
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
