"""Rotations by Euler angles that are not finite: such an angle has no rotation, and
every vector of its item becomes NaN, in either precision, for each of the three
angles and both types; the other items of the batch, and the pair that no rotation
touches (n = 0, or l = 0 of an SH expansion), are what they are without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ITEM, BATCH = 1, 3  # the item with the bad angle


def context(precision):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    ctx.set_precision(precision, 6 if precision else 0)
    return ctx


def angles(which, value):
    e = np.random.default_rng(2).uniform(-3, 3, (BATCH, 3))
    bad = e.copy()
    bad[ITEM, which] = value
    return e, bad


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("rtype", [0, 1])
@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("kind,L,fixed", [("zt", 9, 1), ("st", 40, 1), ("rows", 8, 0)])
def test_rotation(kind, L, fixed, value, which, rtype, precision):
    import zest_gb300 as zg
    n = {"zt": zg.zt_coeff_size, "st": zg.st_coeff_size, "rows": zg.rows_coeff_size}[kind](L)
    c = np.random.default_rng(L).normal(size=(BATCH, n, 2))
    ctx = context(precision)
    got = [getattr(ctx, kind + "_rotate")(c.ravel().copy(), L, e.ravel(), BATCH, rtype).reshape(BATCH, n, 2)
           for e in angles(which, value)]
    ctx.close()
    assert np.isfinite(got[0]).all()
    others = [b for b in range(BATCH) if b != ITEM]
    np.testing.assert_array_equal(got[1][others], got[0][others])
    np.testing.assert_array_equal(got[1][ITEM, :fixed], c[ITEM, :fixed])
    assert np.isnan(got[1][ITEM, fixed:]).all()


@pytest.mark.parametrize("precision", [0, 1])
def test_angle_with_multiples_that_overflow(precision):
    # 2^1022 has finite multiples up to m = 3: vectors of l <= 3 are rotated, the others
    # become NaN (gamma, which every component of a vector depends on)
    import zest_gb300 as zg
    L = 10
    l = np.repeat(np.arange(L), np.arange(1, L + 1))
    ctx = context(precision)
    got = ctx.st_rotate(np.random.default_rng(5).normal(size=(l.size, 2)).ravel(), L,
                        np.array([0.2, 0.5, 2.0 ** 1022])).reshape(-1, 2)
    ctx.close()
    assert np.isfinite(got[l <= 3]).all() and np.isnan(got[l > 3]).all()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_cotangent(value, which, precision):
    import zest_gb300 as zg
    L, n = 12, zg.zt_coeff_size(12)
    rng = np.random.default_rng(7)
    x, y = rng.normal(size=(2, BATCH, n, 2))
    ctx = context(precision)
    got = [ctx.zt_rotate_vjp(x.ravel(), L, e.ravel(), y.ravel(), BATCH)[0].reshape(BATCH, n, 2)
           for e in angles(which, value)]
    ctx.close()
    assert np.isnan(got[1][ITEM, 1:]).all()
    for b in range(BATCH):
        if b != ITEM:
            np.testing.assert_array_equal(got[1][b], got[0][b])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_uneven_batch(which, precision):
    torch = pytest.importorskip("torch")
    import zest_gb300 as zg
    orders = np.array([6, 11, 17])
    cs = [2 * zg.zt_coeff_size(int(L)) for L in orders]
    gs = [int(np.prod(zg.zt_grid_shape(int(L)))) for L in orders]
    c0 = torch.from_numpy(np.random.default_rng(3).normal(size=sum(cs))).cuda()
    ctx = context(precision)
    got = []
    for e in angles(which, np.nan):
        c, g = c0.clone(), torch.zeros(sum(gs), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.zt_rotate_backward_ragged(orders, c, torch.from_numpy(e.ravel()).cuda(), g)
        ctx.synchronize()
        got.append(([v.cpu().numpy() for v in c.split(cs)], [v.cpu().numpy() for v in g.split(gs)]))
    ctx.close()
    assert np.isnan(got[1][0][ITEM][2:]).all()
    assert not np.isfinite(got[1][1][ITEM]).all()
    for b in range(BATCH):
        if b != ITEM:
            np.testing.assert_array_equal(got[1][0][b], got[0][0][b])
            np.testing.assert_array_equal(got[1][1][b], got[0][1][b])
