"""The gathers that keep plane sums between cells (resampling along t, slice
lookup along z), against the oracle bit for bit: several planes per thread
(grids large enough), partial last chunks, and steps along the walked axis of
0, 1, 2 and more source planes, with positions clamped at both ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 4])
@pytest.mark.parametrize("target,source", [
    ((61, 33, 29, 37), (31, 17, 15, 19)),    # refining by about two
    ((61, 33, 29, 37), (33, 19, 15, 2)),     # the smallest t extent
    ((47, 43, 31, 35), (24, 22, 16, 101)),   # several source planes a step
    ((40, 41, 39, 41), (41, 40, 40, 41)),    # one plane a step
    ((5, 4, 3, 2), (9, 8, 7, 6)),            # one plane a thread
])
def test_resample_walk(gpu, orc, nc, target, source):
    import ofblend_gb300 as F
    X, Y, Z, T = source
    rng = np.random.default_rng(3)
    a = rng.standard_normal((T, Z, Y, X, 4) if nc == 4 else (T, Z, Y, X)).astype(np.float32)
    mk = F.Grid4Vec4 if nc == 4 else F.Grid4Real
    for off, scale in [((0, 0, 0, 0), (1, 1, 1, 1)), ((1.0, 0.5, 0.0, 2.0), (0.8, 0.8, 0.8, 0.9))]:
        g = mk(dims=target)
        (F.interpolateGrid4dVec if nc == 4 else F.interpolateGrid4d)(g, mk(dims=source).from_numpy(a),
                                                                    offset=off, scale=scale)
        assert np.array_equal(g.to_numpy(), orc.interpolateGrid4d(target, a, offset=off, scale=scale))


@pytest.mark.parametrize("H,R", [(24, 20), (90, 31), (112, 112), (120, 17)])
def test_lookup_walk(gpu, orc, H, R):
    """1, 1, 2 and 3 cells a thread; 0 to 7 frame cells per slice plane."""
    import ofblend_gb300 as F
    T = 6
    rng = np.random.default_rng(H)
    defo = (rng.standard_normal((T, R, R, R, 4)) * 0.7).astype(np.float32)
    phi = rng.standard_normal((T, H, H, H)).astype(np.float32)
    g = F.Grid4Vec4(dims=(R, R, R, T)).from_numpy(defo)
    gp = F.Grid4Real(dims=(H, H, H, T)).from_numpy(phi)
    dst = F.RealGrid(dims=(H, H, H, 1))
    kw = dict(loadTimeScale=1.0, defoOffset=(0, 0, 0, 0), defoScale=(1, 1, 1, 1),
              defoFactor=(H / R, H / R, H / R, 1.0), overrideSize=(H, H, H, T), bordSkip=3)
    F.loadAdvectTimeSlice_OptInit(7, g)
    F.loadAdvectTimeSlice_OptRun(7, None, dst, gp, 2.5, 0.4, kw["loadTimeScale"], kw["defoOffset"],
                                 kw["defoScale"], kw["defoFactor"], overrideSize=kw["overrideSize"],
                                 bordSkip=kw["bordSkip"])
    F.loadAdvectTimeSlice_Finish(7)
    want = orc.optRunFrame(defo, np.zeros((H, H, H), np.float32), phi, 2.5, 0.4, **kw)
    assert np.array_equal(dst.to_numpy(), np.asarray(want).reshape(H, H, H))
