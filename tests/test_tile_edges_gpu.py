"""FP64 sums at the edges of their tiles: rows, columns and sum lengths around the
tile and warp sizes, every tile shape of the Zernike sums (tuned and by the size
rule) and of the SH sums (column counts 2 to 34), and evaluations of few and odd
points.  Against the oracle at the plain form's bar, 1e-12 relative max-norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def close(got, want):
    return np.max(np.abs(np.ravel(got) - np.ravel(want))) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("tune", [True, False])
@pytest.mark.parametrize("L,Le,batch", [(2, 2, 1), (3, 3, 2), (7, 9, 1), (8, 8, 1), (9, 6, 3), (16, 16, 2), (17, 17, 1),
                                        (31, 31, 1), (33, 33, 2), (49, 49, 1), (64, 50, 1)])
def test_zernike(oracle, L, Le, batch, tune):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    ctx.set_autotune(tune)
    rng = np.random.default_rng(L)
    g = rng.normal(size=(batch,) + zg.zt_grid_shape(L))
    c = ctx.zt_forward(g.ravel(), L, Le, batch).reshape(batch, -1)
    back = ctx.zt_backward(c.ravel(), Le, L, batch).reshape(batch, -1)
    ctx.close()
    for b in range(batch):
        want = oracle.zt_forward(g[b], L, Le, *zg.ZT_GEO)
        assert close(c[b], want)
        assert close(back[b], oracle.zt_backward(want, Le, L, *zg.ZT_GEO))


@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 8, 9, 17])
@pytest.mark.parametrize("L", [3, 17, 40, 131])
def test_sh(oracle, L, batch):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    rng = np.random.default_rng(L + batch)
    g = rng.normal(size=(batch,) + zg.st_grid_shape(L))
    c = ctx.st_forward(g.ravel(), L, batch=batch).reshape(batch, -1)
    back = ctx.st_backward(c.ravel(), L, batch=batch).reshape(batch, -1)
    ctx.close()
    for b in (0, batch - 1):
        want = oracle.st_forward(g[b], L)
        assert close(c[b], want)
        assert close(back[b], oracle.st_backward(want, L))


@pytest.mark.parametrize("nlon,nlat,nrad", [(1, 1, 1), (5, 3, 2), (8, 9, 7), (63, 17, 9), (65, 33, 40)])
def test_evaluate(oracle, nlon, nlat, nrad):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    rng = np.random.default_rng(nlon)
    L, batch = 20, 3
    lon, colat, rad = rng.uniform(0, 6, nlon), rng.uniform(0, 3, nlat), rng.uniform(0, 1, nrad)
    c = rng.normal(size=(batch, zg.zt_coeff_size(L), 2))
    d = rng.normal(size=(batch, zg.st_coeff_size(L), 2))
    v = ctx.zt_evaluate(c.ravel(), L, lon, colat, rad, batch).reshape(batch, -1)
    w = ctx.st_evaluate(d.ravel(), L, lon, colat, batch).reshape(batch, -1)
    ctx.close()
    for b in range(batch):
        assert close(v[b], oracle.zt_evaluate(c[b], L, lon, colat, rad, *zg.ZT_GEO))
        assert close(w[b], oracle.st_evaluate(d[b], L, lon, colat))
