"""Rotations of the split-precision form in 64-bit fixed point: orders around the
warp size and the chunks of the sums (30 pairs of terms), tiles that end within a
batch, all layouts and both types, against the FP64 form at the split form's bar of
1e-11 of each vector's largest coefficient; and exact scaling by powers of two,
vector by vector, since each vector has its own scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def contexts():
    import zest_gb300 as zg
    a, b = zg.Context(0), zg.Context(0)
    b.set_precision(zg.PRECISION_SPLIT, 6)
    return a, b


@pytest.mark.parametrize("rtype", [0, 1])
@pytest.mark.parametrize("kind,L,batch", [
    ("zt", 2, 1), ("zt", 3, 2), ("zt", 9, 3), ("zt", 33, 1), ("zt", 34, 70), ("zt", 62, 2), ("zt", 65, 1),
    ("zt", 130, 1), ("st", 2, 3), ("st", 5, 1), ("st", 33, 9), ("st", 64, 200), ("st", 125, 1), ("st", 256, 1),
    ("st", 257, 1), ("rows", 2, 2), ("rows", 3, 1), ("rows", 40, 3), ("rows", 125, 1)])
def test_against_fp64(kind, L, batch, rtype):
    import zest_gb300 as zg
    fp64, split = contexts()
    n = {"zt": zg.zt_coeff_size, "st": zg.st_coeff_size, "rows": zg.rows_coeff_size}[kind](L)
    rng = np.random.default_rng(3 * L + batch)
    c = rng.normal(size=(batch, n, 2))
    e = rng.uniform(-4, 4, 3 * batch)
    got = [getattr(ctx, kind + "_rotate")(c.ravel().copy(), L, e, batch, rtype).reshape(batch, -1)
           for ctx in (split, fp64)]
    fp64.close()
    split.close()
    assert np.max(np.abs(got[0] - got[1])) <= 1e-11 * np.max(np.abs(got[1]))


def test_scales_and_limits():
    import zest_gb300 as zg
    _, split = contexts()
    rng = np.random.default_rng(8)
    L = 24
    c = rng.normal(size=(zg.st_coeff_size(L), 2))
    l = np.repeat(np.arange(L), np.arange(1, L + 1))
    k = (2.0 ** rng.integers(-250, 250, L))[l][:, None]
    e = np.array([0.3, 1.1, -2.0])
    a = split.st_rotate(c.ravel().copy(), L, e).reshape(-1, 2)
    b = split.st_rotate((c * k).ravel(), L, e).reshape(-1, 2)
    np.testing.assert_array_equal(b[1:], (a * k)[1:])
    # a degree with an infinity or a NaN becomes NaN, a zero one stays zero, the others are as before
    d = c.copy()
    d[l == 7, 0] = np.inf
    d[(l == 9).nonzero()[0][3], 1] = np.nan
    d[l == 11] = 0.0
    f = split.st_rotate(d.ravel(), L, e).reshape(-1, 2)
    bad = (l == 7) | (l == 9)
    assert np.isnan(f[bad]).all() and not f[l == 11].any()
    rest = ~bad & (l != 11)
    np.testing.assert_array_equal(f[rest], a[rest])
    split.close()
