"""When a call on a batch of uneven orders replays a recorded graph, and that it then
gives what an eager one does.  The call that runs a batch for the first time records
it; every call in a row on the same buffers after that is a replay, without a launch of
its own; other buffers, conventions, types, precisions or orders run anew."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def context(precision):
    import zest_gb300 as zg
    ctx = zg.Context(0)
    ctx.set_precision(precision, 6 if precision else 0)
    return ctx


class Batch:
    """Buffers of a batch; fill() gives them new inputs, run() is one call."""

    def __init__(self, orders):
        import zest_gb300 as zg
        self.orders = np.asarray(orders)
        self.coeffs = torch.zeros(sum(2 * zg.zt_coeff_size(int(L)) for L in orders), dtype=torch.float64, device="cuda")
        self.euler = torch.zeros(3 * len(orders), dtype=torch.float64, device="cuda")
        self.grids = torch.zeros(sum(int(np.prod(zg.zt_grid_shape(int(L)))) for L in orders), dtype=torch.float64,
                                 device="cuda")

    def fill(self, seed):
        rng = np.random.default_rng(seed)
        self.coeffs.copy_(torch.from_numpy(rng.normal(size=self.coeffs.numel())))
        self.euler.copy_(torch.from_numpy(rng.uniform(-3, 3, self.euler.numel())))
        self.grids.zero_()
        torch.cuda.synchronize()

    def run(self, ctx, seed, **options):
        """(coefficients, grids, launches of the call)."""
        import zest_gb300 as zg
        self.fill(seed)
        n = zg.launch_count()
        ctx.zt_rotate_backward_ragged(self.orders, self.coeffs, self.euler, self.grids, **options)
        n = zg.launch_count() - n
        ctx.synchronize()
        return self.coeffs.cpu().numpy(), self.grids.cpu().numpy(), n


def expected(precision, orders, seed, **options):
    """The same call, the first of a context."""
    ctx = context(precision)
    c, g, _ = Batch(orders).run(ctx, seed, **options)
    ctx.close()
    return c, g


def check(got, want, scale=1e-13):
    for a, b in zip(got[:2], want):
        assert np.max(np.abs(a - b)) <= scale * np.max(np.abs(b))


ORDERS = [5, 9, 9, 16, 24, 24, 24]


@pytest.mark.parametrize("precision", [0, 1])
def test_calls_in_a_row_are_replays(precision):
    want = [expected(precision, ORDERS, s) for s in range(5)]
    ctx, b = context(precision), Batch(ORDERS)
    for s in range(5):
        got = b.run(ctx, s)
        check(got, want[s])
        assert (got[2] == 0) == (s > 0), (s, got[2])
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_other_buffers(precision):
    want = [expected(precision, ORDERS, s) for s in range(7)]
    ctx, pair = context(precision), [Batch(ORDERS), Batch(ORDERS)]
    for s, which in enumerate([0, 1, 0, 0, 0, 1, 1]):
        got = pair[which].run(ctx, s)
        check(got, want[s])
        assert (got[2] == 0) == (s in (3, 4, 6)), (s, got[2])
    ctx.close()


def test_other_options_on_the_same_buffers():
    import zest_gb300 as zg
    steps = [(0, {}), (0, {}), (0, {"rotation_type": 1}), (0, {"rotation_type": 1}), (0, {"conv": (1, 1, 1)}),
             (0, {"conv": (1, 1, 1)}), (1, {}), (1, {}), (0, {}), (0, {})]
    want = [expected(p, ORDERS, s, **o) for s, (p, o) in enumerate(steps)]
    ctx, b = context(0), Batch(ORDERS)
    for s, (p, o) in enumerate(steps):
        ctx.set_precision(p, 6 if p else 0)
        got = b.run(ctx, s, **o)
        check(got, want[s])
        assert (got[2] == 0) == bool(s & 1), (s, got[2])
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_other_orders(precision):
    lists = [ORDERS, [4, 9, 30], ORDERS]
    want = [expected(precision, o, 10 * i + s) for i, o in enumerate(lists) for s in range(3)]
    ctx = context(precision)
    for i, o in enumerate(lists):
        b = Batch(o)
        for s in range(3):
            got = b.run(ctx, 10 * i + s)
            check(got, want[3 * i + s])
            assert (got[2] == 0) == (s > 0), (i, s, got[2])
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_buffers_freed_between_calls(precision):
    want = [expected(precision, ORDERS, s) for s in range(6)]
    ctx, b = context(precision), Batch(ORDERS)
    for s in range(6):
        if s == 3:
            ctx.trim()
        got = b.run(ctx, s)
        check(got, want[s])
        assert (got[2] == 0) == (s not in (0, 3)), (s, got[2])
    ctx.close()


def test_within_a_capture_of_the_caller():
    # a call on the context's stream while the caller captures it is part of the caller's
    # graph, on buffers that the context has run before and on others
    import zest_gb300 as zg
    stream = torch.cuda.Stream()
    ctx = zg.Context(0, stream.cuda_stream)
    one, two = Batch(ORDERS), Batch(ORDERS)
    want = [expected(0, ORDERS, s) for s in range(4)]
    check(one.run(ctx, 0), want[0])
    check(two.run(ctx, 1), want[1])
    for s, b in ((2, one), (3, two)):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            ctx.zt_rotate_backward_ragged(b.orders, b.coeffs, b.euler, b.grids)
        b.fill(s)
        graph.replay()
        torch.cuda.synchronize()
        check((b.coeffs.cpu().numpy(), b.grids.cpu().numpy()), want[s])
        check(b.run(ctx, 1), want[1])
    ctx.close()
