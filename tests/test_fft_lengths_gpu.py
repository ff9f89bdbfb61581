"""Longitude FFT of every kind of length: prime powers (with and without
twiddles), prime-factor products, small and large direct radices, Rader primes
alone and beside other factors, two Rader candidates, and the multiples of 8 of
the LatLon layout.  The SH transforms through the C-ABI against the oracle's
direct DFT, at the plain form's bar of 1e-12 relative max-norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# LonLat: N = 2 order - 1
LONLAT = [1, 2, 5, 9, 13, 14, 22, 31, 41, 64, 77, 100, 134, 181, 200, 256, 301]
# LatLon: N = 2 order - 1 rounded up to a multiple of 8
LATLON = [1, 4, 5, 20, 33, 44, 45, 64, 100, 172, 200]


@pytest.mark.parametrize("latlon,order", [(0, L) for L in LONLAT] + [(1, L) for L in LATLON])
def test_transform_lengths(oracle, latlon, order):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    batch = 3 if order < 300 else 1  # an odd number of columns, more than one item
    rng = np.random.default_rng(order + 7 * latlon)
    shape = zg.st_grid_shape(order, latlon)
    grids = rng.normal(size=(batch,) + shape)
    c = ctx.st_forward(np.ascontiguousarray(grids).ravel(), order, batch=batch, layout=latlon)
    g = ctx.st_backward(c, order, batch=batch, layout=latlon)
    ctx.close()
    c, g = c.reshape(batch, -1), g.reshape(batch, -1)
    for b in range(batch):
        ref = oracle.st_forward(grids[b], order, latlon=bool(latlon))
        back = oracle.st_backward(ref, order, latlon=bool(latlon)).ravel()
        assert np.max(np.abs(c[b] - ref.ravel())) <= 1e-12 * np.max(np.abs(ref))
        assert np.max(np.abs(g[b] - back)) <= 1e-12 * np.max(np.abs(back))
