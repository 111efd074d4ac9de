"""Deformation solves whose coarse levels come down to one cell along an axis.
Such a level has no interior, so it returns the velocity that it is given."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(wSmooth=0.001, wEnergy=0.0001, cgAccuracy=0.01, cfl=999, multiStep=3, doFinalProject=False)


def pair(dims):
    rng = np.random.default_rng(sum(dims))
    X, Y, Z, T = dims
    base = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
    for ax in range(4):  # a smooth field of the solver's input magnitude
        base = (base + np.roll(base, 1, ax)).astype(np.float32) * np.float32(0.5)
    i0 = base * np.float32(0.02)
    return i0, np.roll(i0, 1, axis=3) + np.float32(0.001)


# (X, Y, Z, T), minGridSize: an axis of 3 halves to 1, and stays there where the
# level above it is halved once more
@pytest.mark.parametrize("dims,mn", [((24, 24, 24, 3), 12), ((24, 24, 3, 24), 12), ((24, 3, 24, 24), 12),
                                     ((3, 24, 24, 24), 1), ((40, 24, 24, 3), 10), ((40, 3, 24, 3), 5)])
def test_thin_levels_add_nothing(dims, mn):
    import ofblend_gb300 as F

    i0, i1 = pair(dims)
    g0, g1 = F.Grid4Real(dims=dims).from_numpy(i0), F.Grid4Real(dims=dims).from_numpy(i1)
    out = []
    for size in (mn, 9999):  # with the thin levels below, and the finest level alone
        v = F.Grid4Vec4(dims=dims)
        err = F.opticalFlowMultiscale4d(v, g0, g1, minGridSize=size, postVelBlur=4, resetBndWidth=0.01, **KW)
        out.append((err, v.to_numpy()))
    assert out[0][0] == out[1][0] and out[1][1].any()
    assert np.array_equal(out[0][1], out[1][1])


def axis_matrix(nt, ns):
    """interpolGridTempl's weights along an axis (optflow4d.cpp:40-57) in FP64."""
    m = np.zeros((nt, ns))
    for i in range(nt):
        p = max(i * (ns / nt) + 0.5 * ns / nt - 0.5, 0.0)
        b = min(int(p), ns - 1)
        m[i, b] += 1.0 - (p - b) if b + 1 < ns else 1.0
        if b + 1 < ns:
            m[i, b + 1] += p - b
    return m


def resample(v, shape):
    for ax, n in enumerate(shape):
        v = np.moveaxis(np.tensordot(axis_matrix(n, v.shape[ax]), v, (1, ax)), 0, ax)
    return v


@pytest.mark.parametrize("dims,levels", [((22, 18, 14, 2), 1), ((44, 18, 14, 2), 2), ((22, 2, 14, 6), 1),
                                         ((22, 14, 2, 6), 1), ((2, 14, 18, 6), 1)])
def test_velocity_through_thin_levels(dims, levels):
    """No level has an interior: the input velocity comes back restricted and
    prolonged again."""
    import ofblend_gb300 as F

    i0, i1 = pair(dims)
    rng = np.random.default_rng(3)
    vel = rng.standard_normal(i0.shape + (4,)).astype(np.float32)
    v = F.Grid4Vec4(dims=dims).from_numpy(vel)
    F.opticalFlowMultiscale4d(v, F.Grid4Real(dims=dims).from_numpy(i0), F.Grid4Real(dims=dims).from_numpy(i1),
                              minGridSize=dims[0] // 2 ** levels, **KW)
    shapes = [i0.shape]
    for _ in range(levels):
        shapes.append(tuple(max(n // 2, 1) for n in shapes[-1]))
    want = vel.astype(np.float64)
    for s in shapes[1:] + shapes[-2::-1]:
        want = resample(want, s)
    # a resampled value is a weighted mean of at most 16 with some 20 roundings on
    # its way, of values below 6; 2 x levels resamplings
    assert np.abs(v.to_numpy() - want).max() <= 2 * levels * 20 * 2.0 ** -24 * 6
