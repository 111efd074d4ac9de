"""The direct Gaussian blur's tile shapes (32, 16 and 8 columns; 8 and 4 rows a
thread; one to four warps; several y tiles) against its plain-load counterpart,
which test_gpu_parity.py holds to the oracle: bit for bit, zeros' signs
included, on grids whose extents leave partial tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(64, 64, 20, 20), (48, 48, 24, 24), (40, 41, 30, 30), (33, 70, 26, 25),
                                  (24, 24, 24, 16), (8, 130, 9, 7), (17, 5, 6, 9), (2, 3, 4, 5)])
@pytest.mark.parametrize("sigma", [2.0, 1.0])
def test_blur_tiles_match_plain_loads(dims, sigma):
    import ofblend_gb300 as F
    from ofblend_gb300 import _lib
    ctx = F.Context(0)
    X, Y, Z, T = dims
    rng = np.random.default_rng(X * Y)
    a = rng.standard_normal((T, Z, Y, X, 4)).astype(np.float32)
    a[rng.random(a.shape) < 0.3] = 0.0
    a[..., 1] *= np.float32(-0.0)  # a component of signed zeros
    a[..., 2] *= np.float32(1e-30)
    got = []
    for tma in (0, 1):
        ctx.set_option(_lib.FLOF_OPT_SLAB_TMA, tma)
        g = F.Grid4Vec4(dims=dims, ctx=ctx).from_numpy(a)
        F.gaussianBlur4d(g, sigma)
        got.append(g.to_numpy().view(np.uint32))
    assert np.array_equal(got[0], got[1])
