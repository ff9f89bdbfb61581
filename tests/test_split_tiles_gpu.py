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


@pytest.mark.parametrize("ka", [(0,), (-500, 0, 40), (-900, -500, -30, 0, 500, 900)])
def test_row_scales_are_exact(ctx, ka):
    # rows scaled by powers of two: warps whose results all stay in the normal
    # range, and warps with some below it (which are 0) or above (infinite).
    # The integer sums are exact as above, and so are the scaled ones.
    import zest_gb300
    M, N, K = 260, 50, 40
    rng = np.random.default_rng(len(ka))
    A = rng.integers(-(1 << 12) + 1, 1 << 12, size=(M, K)).astype(np.float64)
    B = rng.integers(-(1 << 12) + 1, 1 << 12, size=(N, K)).astype(np.float64)
    A[7] = 0.0
    ea = np.array([ka[i % len(ka)] for i in range(M)])
    eb = np.array([(0, 300, -450)[i % 3] if len(ka) > 1 else 0 for i in range(N)])
    ctx.set_precision(zest_gb300.PRECISION_SPLIT, 6)
    try:
        C = ctx.split_gemm(np.ldexp(A, ea[:, None]), np.ldexp(B, eb[:, None]))
    finally:
        ctx.set_precision(zest_gb300.PRECISION_FP64)
    with np.errstate(over="ignore"):
        ref = np.ldexp(A @ B.T, ea[:, None] + eb[None, :])
    ref[np.abs(ref) < 2.0 ** -1022] = 0.0
    assert np.array_equal(C, ref)
