"""Longitude transforms of the split-precision path in 64-bit fixed point: every
kind of length (prime powers, prime-factor products, direct and Rader radices,
LatLon multiples of 8), an odd number of columns, truncation both ways, against the
FP64 form at the split form's bar of 1e-11; and exact scaling by powers of two,
column by column, since each column has its own scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def contexts():
    import zest_gb300 as zg
    a, b = zg.Context(0), zg.Context(0)
    b.set_precision(zg.PRECISION_SPLIT, 6)
    return a, b


def close(x, y):
    return np.max(np.abs(x - y)) <= 1e-11 * np.max(np.abs(y))


@pytest.mark.parametrize("latlon,L,Le,batch", [
    (0, 2, 2, 1), (0, 3, 3, 3), (0, 5, 4, 2), (0, 9, 11, 1), (0, 13, 13, 1), (0, 14, 14, 2), (0, 22, 22, 1),
    (0, 64, 50, 3), (0, 77, 77, 1), (0, 100, 100, 5), (0, 181, 200, 1), (0, 260, 260, 2), (0, 301, 301, 1),
    (0, 1011, 1011, 1), (1, 3, 3, 1), (1, 20, 20, 3), (1, 33, 40, 1), (1, 45, 45, 2), (1, 172, 150, 1),
    (1, 257, 257, 1)])
def test_against_fp64(latlon, L, Le, batch):
    import zest_gb300 as zg
    fp64, split = contexts()
    rng = np.random.default_rng(L)
    g = rng.normal(size=batch * int(np.prod(zg.st_grid_shape(L, latlon))))
    c = [ctx.st_forward(g, L, Le, batch, layout=latlon) for ctx in (split, fp64)]
    b = [ctx.st_backward(c[1], Le, L, batch, layout=latlon) for ctx in (split, fp64)]
    fp64.close()
    split.close()
    assert close(*c)
    assert close(*b)


@pytest.mark.parametrize("L,batch", [(258, 1), (270, 2)])
def test_zernike_above_256(L, batch):
    import zest_gb300 as zg
    torch = pytest.importorskip("torch")
    fp64, split = contexts()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(L)
    c0 = torch.randn(batch * 2 * zg.zt_coeff_size(L), dtype=torch.float64, device="cuda", generator=gen)
    g = fp64.zt_backward(c0, L, batch=batch)
    gs = split.zt_backward(c0, L, batch=batch)
    assert float((g - gs).abs().max()) <= 1e-11 * float(g.abs().max())
    c, cs = fp64.zt_forward(g, L, batch=batch), split.zt_forward(g, L, batch=batch)
    assert float((c - cs).abs().max()) <= 1e-11 * float(c.abs().max())
    fp64.close()
    split.close()


def test_scales():
    import zest_gb300 as zg
    _, split = contexts()
    rng = np.random.default_rng(5)
    L, batch = 40, 3
    g = rng.normal(size=(batch, int(np.prod(zg.st_grid_shape(L)))))
    k = 2.0 ** np.array([[-300.0], [0.0], [250.0]])
    c = split.st_forward(g.ravel(), L, batch=batch).reshape(batch, -1)
    s = split.st_forward((g * k).ravel(), L, batch=batch).reshape(batch, -1)
    np.testing.assert_array_equal(s, c * k)
    split.close()
