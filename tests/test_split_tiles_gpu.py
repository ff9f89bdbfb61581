"""Column tiles of the split GEMMs: every unit is as wide as its valid columns
rounded up to 16, and units of mixed widths follow one another in a CTA.

Integer operands below 2^12 have only their two leading digits, whose products
(levels 0 to 2) are kept by every slice count, and sums of 96 products stay
below 2^31: the product is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import zest_gb300
    from zest_gb300 import build
    build.build()
    c = zest_gb300.Context(0)
    yield c
    c.close()


# 8 + 128 * 170 rows: at least 171 row tiles, so that the CTAs take several
# units each and change sides and widths between them
@pytest.mark.parametrize("S", [4, 5, 6])
@pytest.mark.parametrize("N", [1, 16, 17, 32, 33, 48, 49, 64, 65, 80, 81, 97, 113, 129, 192, 200])
def test_tile_widths_are_exact(ctx, S, N):
    import zest_gb300
    M, K = 8 + 128 * 170, (96, 24, 10)[N % 3]
    rng = np.random.default_rng(100 * S + N)
    A = rng.integers(-(1 << 12) + 1, 1 << 12, size=(M, K)).astype(np.float64)
    B = rng.integers(-(1 << 12) + 1, 1 << 12, size=(N, K)).astype(np.float64)
    ctx.set_precision(zest_gb300.PRECISION_SPLIT, S)
    try:
        C = ctx.split_gemm(A, B)
    finally:
        ctx.set_precision(zest_gb300.PRECISION_FP64)
    assert np.array_equal(C, A @ B.T)
