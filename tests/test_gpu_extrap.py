"""extrap4dLsSimple's bit-mask fronts at the row lengths where a row's words
change (one cell inside, either side of 32 and 64 cells) and on the smallest
extents, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inside", [False, True])
@pytest.mark.parametrize("dims", [(3, 3, 3, 3), (4, 9, 7, 5), (31, 6, 5, 4), (32, 5, 6, 4), (33, 6, 4, 7),
                                  (34, 5, 5, 5), (64, 4, 6, 5), (65, 7, 5, 4), (66, 5, 8, 6)])
def test_extrap_row_lengths(gpu, orc, dims, inside):
    import ofblend_gb300 as F
    X, Y, Z, T = dims
    rng = np.random.default_rng(X * 100 + T)
    a = rng.standard_normal((T, Z, Y, X)).astype(np.float32)
    sign = -1.0 if inside else 1.0
    a = (sign * np.abs(a)).astype(np.float32)
    # a few seeds of the region, some on the row's first and last inner cells
    for x in {1, X // 2, X - 2}:
        a[T // 2, Z // 2, Y // 2, x] *= -1.0
    for distance in (0, 1, 2, 12):
        want = orc.extrap4dLsSimple(a, distance, inside)
        g = F.Grid4Real(dims=dims).from_numpy(a)
        F.extrap4dLsSimple(g, distance, inside)
        assert np.array_equal(g.to_numpy(), want)
