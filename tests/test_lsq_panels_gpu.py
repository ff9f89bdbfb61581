"""Least-squares fits at the edges of the QR's panels and tiles: unknowns around
the panel width (32) and the column tiles, points from the unknowns on (square
systems) and around the rows of a block, one and many data vectors, and more
points than the panels keep in shared memory.  Against numpy's least-squares
solution of the oracle's design matrix; both are backward stable, so they agree
within cond(A) times a few hundred roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,points,batch", [(1, 1, 1), (1, 70, 2), (2, 4, 1), (5, 25, 3), (5, 63, 1), (5, 129, 1),
                                            (6, 37, 2), (6, 300, 31), (6, 130000, 2), (8, 64, 1), (8, 1000, 33),
                                            (9, 82, 1), (17, 2500, 1), (17, 9900, 16)])
def test_fit(oracle, L, points, batch):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    rng = np.random.default_rng(points + L)
    lat, lon = np.arcsin(rng.uniform(-1, 1, points)), rng.uniform(0, 2 * np.pi, points)
    P = oracle.plm_real(L, 0, 0, np.sin(lat)).reshape(-1, points)
    cols, at = [], []
    for l in range(L):
        for m in range(l + 1):
            for c in range(2 if m else 1):
                cols.append(P[l * (l + 1) // 2 + m] * (np.sin(m * lon) if c else np.cos(m * lon)))
                at.append(2 * (l * (l + 1) // 2 + m) + c)
    A = np.stack(cols, 1)
    d = rng.normal(size=(batch, points))
    got = ctx.st_lsq(d.ravel(), L, lat, lon, batch).reshape(batch, -1)
    ctx.close()
    x, _, _, sv = np.linalg.lstsq(A, d.T, rcond=None)
    bound = 500 * 2.0 ** -53 * sv[0] / sv[-1] * np.linalg.norm(d) / sv[-1]
    assert np.max(np.abs(got[:, at] - x.T)) <= bound
    rest = np.ones(got.shape[1], bool)
    rest[at] = False
    assert not got[:, rest].any()
