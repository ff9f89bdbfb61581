"""FP64 rotations in tiles of one degree: orders around the warp size, batches that
give every vector count per thread (2, 4, 8) and end within a tile, all layouts,
against the oracle at the plain form's bar of 1e-12 relative max-norm.  The
gradient kernel's coefficient cotangent is the inverse rotation (1e-13: the same
products, two roundings apart), its angle gradients agree with central
differences (h = 1e-6, 1e-7 of their size plus the rounding of the loss)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vectors(rng, kind, L, batch):
    import zest_gb300 as zg
    n = {"zt": zg.zt_coeff_size, "st": zg.st_coeff_size, "rows": zg.rows_coeff_size}[kind](L)
    return rng.normal(size=(batch, n, 2))


@pytest.mark.parametrize("rtype", [0, 1])
@pytest.mark.parametrize("L,batch", [(2, 1), (3, 5), (9, 2), (31, 1), (33, 3), (33, 100), (33, 201), (65, 2), (90, 1)])
@pytest.mark.parametrize("kind", ["zt", "st"])
def test_rotate(oracle, kind, L, batch, rtype):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    rng = np.random.default_rng(L * 7 + batch)
    c = vectors(rng, kind, L, batch)
    e = rng.uniform(-4, 4, (batch, 3))
    rotate, ref = ((ctx.zt_rotate, oracle.zt_rotate) if kind == "zt" else (ctx.st_rotate, oracle.st_rotate))
    got = rotate(c.ravel().copy(), L, e.ravel(), batch, rtype).reshape(c.shape)
    ctx.close()
    for b in {0, batch // 2, batch - 1}:
        want = ref(c[b].copy(), L, e[b], rtype)
        assert np.max(np.abs(got[b].ravel() - np.ravel(want))) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("rtype", [0, 1])
@pytest.mark.parametrize("L,batch", [(2, 1), (3, 4), (17, 2), (33, 3), (33, 120), (70, 1)])
@pytest.mark.parametrize("kind", ["zt", "st"])
def test_gradients(kind, L, batch, rtype):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    rng = np.random.default_rng(L * 5 + batch)
    x, y = vectors(rng, kind, L, batch), vectors(rng, kind, L, batch)
    e = rng.uniform(-4, 4, (batch, 3))
    rotate, vjp = ((ctx.zt_rotate, ctx.zt_rotate_vjp) if kind == "zt" else (ctx.st_rotate, ctx.st_rotate_vjp))
    xb, eb = vjp(x.ravel(), L, e.ravel(), y.ravel(), batch, rtype)
    alone, _ = vjp(x.ravel(), L, e.ravel(), y.ravel(), batch, rtype, want_euler=False)
    _, angles = vjp(x.ravel(), L, e.ravel(), y.ravel(), batch, rtype, want_coeffs=False)
    assert np.max(np.abs(xb - alone)) <= 1e-13 * np.max(np.abs(alone))
    np.testing.assert_array_equal(eb, angles)
    h = 1e-6
    size = np.linalg.norm(x.reshape(batch, -1), axis=1) * np.linalg.norm(y.reshape(batch, -1), axis=1)
    for k in range(3):
        d = []
        for s in (h, -h):
            f = e.copy()
            f[:, k] += s
            d.append((rotate(x.ravel().copy(), L, f.ravel(), batch, rtype).reshape(batch, -1) *
                      y.reshape(batch, -1)).sum(1))
        fd = (d[0] - d[1]) / (2 * h)
        assert np.all(np.abs(fd - eb.reshape(batch, 3)[:, k]) <= 1e-7 * size)
    ctx.close()
