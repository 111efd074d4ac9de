"""The velocity blurs compute only what the cells that survive the border reset
depend on: whole solves and projections with a reset border, whose intermediate
buffers start from arbitrary pool memory, against the plain-load kernels, which
blur every cell: bit for bit (blurType 1), with border widths from one cell to
more than the grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [0.001, 0.1, 0.3, 0.49, 0.7])
@pytest.mark.parametrize("dims", [(26, 23, 21, 17), (41, 12, 9, 22)])
def test_reset_border_blurs(orc, width, dims):
    import ofblend_gb300 as F
    from ofblend_gb300 import _lib, synth
    ctx = F.Context(0)
    X, Y, Z, T = dims
    i0 = synth.flow_input(synth.scene_for(0), dims)
    i1 = synth.flow_input(synth.scene_for(1), dims)
    # leave NaN in the pool's buffers of this size
    junk = F.Grid4Vec4(dims=dims, ctx=ctx).from_numpy(np.full((T, Z, Y, X, 4), np.nan, np.float32))
    F.gaussianBlur4d(junk, 2.0)
    F.gaussianBlur4d(junk, 2.0, 2)
    g0 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i0)
    g1 = F.Grid4Real(dims=dims, ctx=ctx).from_numpy(i1)
    rng = np.random.default_rng(7)
    v0 = (rng.standard_normal((T, Z, Y, X, 4)) * 0.8).astype(np.float32)
    got = {}
    for tma in (0, 1):
        ctx.set_option(_lib.FLOF_OPT_SLAB_TMA, tma)
        v = F.Grid4Vec4(dims=dims, ctx=ctx)
        F.opticalFlow4d(v, g0, g1, wSmooth=0.001, wEnergy=0.0001, postVelBlur=4.0, cgAccuracy=1e-2,
                        resetBndWidth=width)
        w = F.Grid4Vec4(dims=dims, ctx=ctx).from_numpy(v0)
        d = F.Grid4Vec4(dims=dims, ctx=ctx)
        F.corrVelsOf4d(d, w, g0, None, g1, threshPhi=4.0, postVelBlur=4.0, resetBndWidth=width, maxIter=40)
        got[tma] = [a.to_numpy() for a in (v, w, d)]
    for a, b in zip(got[0], got[1]):
        assert np.array_equal(a, b)
    # blurType 2 against blurType 1: equal up to rounding, finite everywhere
    s = F.Grid4Vec4(dims=dims, ctx=ctx)
    F.opticalFlow4d(s, g0, g1, wSmooth=0.001, wEnergy=0.0001, postVelBlur=4.0, cgAccuracy=1e-2, blurType=2,
                    resetBndWidth=width)
    a, b = s.to_numpy(), got[1][0]
    assert np.isfinite(a).all()
    assert np.linalg.norm(a - b) <= 1e-5 * max(np.linalg.norm(b), 1e-30)
