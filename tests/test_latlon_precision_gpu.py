"""Longitude transforms of LatLon grids run in FP64 in both precisions.  A field with
a large mean and small variations shows it: what the transform loses beside the mean
is a large part of the variations.

Lengths N = 4^k whose sums have no rounding at the size of the mean make the bounds
sharp.  Forward: the grid is 1 + d with d a multiple of 2^-(52 - 2k), so that sums of
N of its values are exact in FP64 and the orders m > 0 are rounded at their own size;
they have to agree with the FP64 form to 1e-11 of the largest, the bar of the split
Legendre sums.  Backward: the mean is 2^20 exactly, so a value passes through k stages
of two roundings of at most 2^-33, in either precision; the sums of the variations
(below 2^10) differ by less than one more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LATLON = 1


def contexts():
    import zest_gb300 as zg
    a, b = zg.Context(0), zg.Context(0)
    b.set_precision(zg.PRECISION_SPLIT, 6)
    return a, b


@pytest.mark.parametrize("L,k,batch", [(32, 3, 3), (127, 4, 2), (512, 5, 1)])
def test_forward_variations_beside_the_mean(L, k, batch):
    import zest_gb300 as zg
    shape = zg.st_grid_shape(L, LATLON)
    assert shape[1] == 4 ** k
    rng = np.random.default_rng(L)
    g = 1.0 + rng.integers(-2 ** 12, 2 ** 12, size=(batch, *shape)) * 2.0 ** (2 * k - 52)
    fp64, split = contexts()
    want, got = (ctx.st_forward(g.ravel(), L, batch=batch, layout=LATLON).reshape(batch, -1, 2) for ctx in (fp64, split))
    fp64.close()
    split.close()
    m = np.concatenate([np.arange(l + 1) for l in range(L)])
    assert np.max(np.abs(got - want)[:, m > 0]) <= 1e-11 * np.max(np.abs(want[:, m > 0]))


@pytest.mark.parametrize("L,k,batch", [(128, 4, 2), (511, 5, 1)])
def test_backward_variations_beside_the_mean(L, k, batch):
    import zest_gb300 as zg
    shape = zg.st_grid_shape(L, LATLON)
    assert shape[1] == 4 ** k
    rng = np.random.default_rng(L)
    m = np.concatenate([np.arange(l + 1) for l in range(L)])
    l = np.repeat(np.arange(L), np.arange(1, L + 1))
    c = rng.uniform(-1, 1, size=(batch, l.size, 2)) / (l[:, None] + 1.0)
    c[:, m == 0] = 0.0
    c[:, 0, 0] = 2.0 ** 20
    fp64, split = contexts()
    want, got = (ctx.st_backward(c.ravel(), L, batch=batch, layout=LATLON) for ctx in (fp64, split))
    fp64.close()
    split.close()
    assert np.max(np.abs(want - 2.0 ** 20)) < 2.0 ** 10
    assert np.max(np.abs(got - want)) <= (2 * 2 * k + 1) * 2.0 ** -33
