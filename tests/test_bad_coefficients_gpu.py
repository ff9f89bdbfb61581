"""Rotations of expansions whose unused entries (the sine parts of m = 0) are not
finite: the vector becomes NaN in either precision, as it does for every other entry,
and the others are what they are without it; a finite entry there changes nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e200])
def test_sine_part_of_order_zero(value, precision):
    import zest_gb300 as zg
    L = 20
    l = np.repeat(np.arange(L), np.arange(1, L + 1))
    c = np.random.default_rng(4).normal(size=(l.size, 2))
    c[l * (l + 1) // 2, 1] = 0.0
    d = c.copy()
    d[(l == 6).nonzero()[0][0], 1] = value
    ctx = zg.Context(0)
    ctx.set_precision(precision, 6 if precision else 0)
    e = np.array([0.4, 1.3, -0.7])
    a, b = (ctx.st_rotate(x.ravel().copy(), L, e).reshape(-1, 2) for x in (c, d))
    ctx.close()
    if np.isfinite(value):
        np.testing.assert_array_equal(b, a)
    else:
        assert np.isnan(b[l == 6]).all()
        np.testing.assert_array_equal(b[l != 6], a[l != 6])
