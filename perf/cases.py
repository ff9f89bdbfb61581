"""The work that users of this framework have it do, as cases that can be timed.

listed() gives the cases, draw(rng) one more case of the same ranges,
prepare(case, seed) the inputs a program holds before its call, run(state) one
pass through the public entry points, work(case) the bytes and operations that
a pass cannot do without and exact(case, seed) the outputs of a pass computed
in 64 bits by torch and numpy alone.

The families (a case's "op"):
  zt        Zernike transforms of a batch of functions on ball grids: forward,
            backward, both in turn ("round"), or forward and its adjoint ("vjp")
  st        spherical-harmonic transforms, LonLat or LatLon grids: the same
  rotate    Rotor::rotate of a batch of expansions, on its own or with the
            gradients of coefficients and Euler angles
  ragged    expansions of different orders, each rotated and synthesised
  evaluate  expansions evaluated at arbitrary points (the grid evaluator)
  lsq       least-squares fits of expansions to data at scattered points
  spectra   power spectra of a batch of expansions
"precision" is the context's: "fp64" (the default form) or "split" (six BF16
slices on the tensor cores).  "conv" is the index of a convention triple.
"""
import math

import numpy as np
import torch

import zest_gb300 as zg


def listed():
    return [
        # a single small function, there and back: latency and launches
        {"name": "zt_fp64_20x1", "op": "zt", "precision": "fp64", "mode": "round", "order": 20, "exp_order": 20,
         "batch": 1, "conv": 4},
        # a differentiable layer of a fit: coefficients of 32 functions and the grid cotangents, default precision
        {"name": "zt_fp64_vjp_100x32", "op": "zt", "precision": "fp64", "mode": "vjp", "order": 100,
         "exp_order": 100, "batch": 32, "conv": 4},
        # the benchmark's batch: analysis and synthesis of 64 functions at order 200 on the tensor cores
        {"name": "zt_split_200x64", "op": "zt", "precision": "split", "mode": "round", "order": 200,
         "exp_order": 200, "batch": 64, "conv": 4},
        # synthesis of expansions on a coarser grid than their order, odd sizes, unnormed with the phase
        {"name": "zt_split_back_63x17", "op": "zt", "precision": "split", "mode": "backward", "order": 63,
         "exp_order": 80, "batch": 17, "conv": 7},
        # global models of the sphere at lmax 1023, plain FP64
        {"name": "st_fp64_1024x8", "op": "st", "precision": "fp64", "mode": "round", "order": 1024,
         "exp_order": 1024, "batch": 8, "conv": 0, "latlon": False},
        # the same on the tensor cores
        {"name": "st_split_1024x8", "op": "st", "precision": "split", "mode": "round", "order": 1024,
         "exp_order": 1024, "batch": 8, "conv": 0, "latlon": False},
        # rotational alignment: rotate 256 expansions, then the gradients of a loss
        {"name": "rotate_fp64_grad_64x256", "op": "rotate", "precision": "fp64", "kind": "zt", "grad": True,
         "order": 64, "batch": 256, "type": 0},
        # plain rotation of the same batch on the tensor cores
        {"name": "rotate_split_64x256", "op": "rotate", "precision": "split", "kind": "zt", "grad": False,
         "order": 64, "batch": 256, "type": 0},
        # a catalogue of expansions of uneven order, rotated and synthesised
        {"name": "ragged_split_1024", "op": "ragged", "precision": "split", "items": 1024, "lo": 8, "hi": 128},
        # values of 8 models at a product grid of arbitrary points
        {"name": "evaluate_100x8", "op": "evaluate", "precision": "fp64", "kind": "zt", "order": 100, "batch": 8,
         "nlon": 200, "nlat": 100, "nrad": 100},
        # fits to 20,000 scattered observations, 16 data vectors at the same points
        {"name": "lsq_st_32x16", "op": "lsq", "precision": "fp64", "kind": "st", "order": 32, "points": 20000,
         "batch": 16},
        # the spectra of the models above
        {"name": "spectra_st_1024x8", "op": "spectra", "precision": "fp64", "kind": "st", "order": 1024, "batch": 8},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["zt", "zt", "zt", "st", "st", "rotate", "rotate", "ragged", "evaluate", "lsq", "spectra"])
    if op == "zt":
        precision = rng.choice(["fp64", "split"])
        order = _log_int(rng, 6, 200)
        # at most 64 functions, and no more work than the listed cases of the precision
        most = 64 if precision == "split" else int(min(64, 100 ** 4 * 32 / order ** 4))
        mode = rng.choice(["round", "forward", "backward", "vjp"])
        exp = order if rng.random() < 0.6 else max(4, int(order * rng.uniform(0.6, 1.3)))
        return {"op": op, "precision": precision, "mode": mode, "order": order,
                "exp_order": order if mode == "vjp" else exp, "batch": _log_int(rng, 1, max(1, most)),
                "conv": rng.randrange(8)}
    if op == "st":
        precision = rng.choice(["fp64", "split"])
        order = _log_int(rng, 8, 1024)
        mode = rng.choice(["round", "forward", "backward", "vjp"])
        exp = order if rng.random() < 0.6 else max(4, min(1024, int(order * rng.uniform(0.6, 1.3))))
        return {"op": op, "precision": precision, "mode": mode, "order": order,
                "exp_order": order if mode == "vjp" else exp,
                "batch": _log_int(rng, 1, int(min(64, max(1, 8 * (1024 / order) ** 3)))), "conv": rng.randrange(4),
                "latlon": rng.random() < 0.4}
    if op == "rotate":
        kind = rng.choice(["zt", "st"])
        order = _log_int(rng, 4, 100 if kind == "zt" else 200)
        cost = order ** 4 if kind == "zt" else 3 * order ** 3
        return {"op": op, "precision": rng.choice(["fp64", "split"]), "kind": kind, "grad": rng.random() < 0.4,
                "order": order, "batch": _log_int(rng, 1, max(1, int(min(1024, 64 ** 4 * 256 / cost)))),
                "type": rng.randrange(2)}
    if op == "ragged":
        lo = rng.randrange(8, 40)
        return {"op": op, "precision": rng.choice(["split", "split", "fp64"]), "items": _log_int(rng, 8, 256),
                "lo": lo, "hi": rng.randrange(lo + 1, 129)}
    if op == "evaluate":
        kind = rng.choice(["zt", "st"])
        order = _log_int(rng, 6, 100)
        return {"op": op, "precision": "fp64", "kind": kind, "order": order, "batch": _log_int(rng, 1, 8),
                "nlon": _log_int(rng, 10, 200), "nlat": _log_int(rng, 10, 100), "nrad": _log_int(rng, 10, 100)}
    if op == "lsq":
        kind = rng.choice(["st", "zt"])
        order = _log_int(rng, 4, 28 if kind == "st" else 11)
        unknowns = order * order if kind == "st" else order * (order + 1) * (order + 2) // 6
        return {"op": op, "precision": "fp64", "kind": kind, "order": order,
                "points": unknowns + _log_int(rng, max(64, unknowns), 18000), "batch": _log_int(rng, 1, 16)}
    kind = rng.choice(["st", "zt"])
    order = _log_int(rng, 16, 1024 if kind == "st" else 200)
    return {"op": op, "precision": "fp64", "kind": kind, "order": order, "batch": _log_int(rng, 1, 8)}


# ---- sizes and layouts ---------------------------------------------------------
def _zt_conv(case):
    c = case["conv"]
    return (c >> 2, (c >> 1) & 1, c & 1)  # Zernike norm (1 unnormed), SH norm (1 quantum mechanics), phase (1 CS)


def _st_conv(case):
    c = case["conv"]
    return (c >> 1, c & 1)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _orders(case):
    """The orders of a catalogue: the same ones pass for pass, with other coefficients and rotations."""
    rng = np.random.default_rng(4096)
    return np.sort(rng.integers(case["lo"], case["hi"] + 1, size=case["items"])).astype(np.int32)


def _zt_index(L):
    """(n, l, m) of every coefficient pair of a Zernike expansion, in its order."""
    n, l, m = [], [], []
    for nn in range(L):
        ls = np.arange(nn & 1, nn + 1, 2)
        ll = np.repeat(ls, ls + 1)
        l.append(ll)
        m.append(np.concatenate([np.arange(x + 1) for x in ls]))
        n.append(np.full(ll.size, nn))
    return np.concatenate(n), np.concatenate(l), np.concatenate(m)


def _st_index(L):
    """(l, m) of every coefficient pair of an SH expansion, in its order."""
    l = np.repeat(np.arange(L), np.arange(1, L + 1))
    return l, np.concatenate([np.arange(x + 1) for x in range(L)])


def _gl(n):
    """Gauss-Legendre nodes (ascending) and weights by Newton's method in extended precision."""
    f = np.longdouble
    i = np.arange(n, dtype=f)
    x = -np.cos(np.asarray(np.pi, dtype=f) * (i + f(0.75)) / (f(n) + f(0.5)))
    for _ in range(4):
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / f(k)
        if n == 1:
            p0, p1 = np.ones_like(x), x
        dp = n * (x * p1 - p0) / (x * x - 1)
        x = x - p1 / dp
    w = 2 / ((1 - x * x) * dp * dp)
    return x.astype(np.float64), w.astype(np.float64)


# ---- inputs ----------------------------------------------------------------------
_held = {}  # the context of the case at hand, as a program keeps one


def _context(case):
    key = tuple(sorted((k, str(v)) for k, v in case.items()))
    if _held.get("key") != key:
        _held.clear()
        ctx = zg.Context(0)
        if case["precision"] == "split":
            ctx.set_precision(zg.PRECISION_SPLIT, 6)
        _held.update(key=key, ctx=ctx)
    return _held["ctx"]


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(1000 + seed)
    return g


def _zt_scale(L):
    """(n+1)^-1.5 per value, 0 for the sine part of m = 0."""
    n, _, m = _zt_index(L)
    s = np.stack([(n + 1.0) ** -1.5, np.where(m > 0, (n + 1.0) ** -1.5, 0.0)], 1)
    return torch.from_numpy(s.ravel()).to(_device())


def _st_scale(L):
    l, m = _st_index(L)
    s = np.stack([(l + 1.0) ** -1.0, np.where(m > 0, (l + 1.0) ** -1.0, 0.0)], 1)
    return torch.from_numpy(s.ravel()).to(_device())


def _coefficients(scale, batch, gen):
    """`batch` expansions of random coefficients that fall with the degree."""
    c = torch.randn(batch, scale.numel(), dtype=torch.float64, device=scale.device, generator=gen)
    return (c * scale).reshape(-1)


def _blobs(lon, lat_sin, rad, batch, gen, order):
    """Functions sampled on a grid [b] + `order`: two Gaussian blobs each and 1% of noise."""
    dev = _device()
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    lon, z, r = t(lon), t(lat_sin), t(rad)
    c = torch.rand(batch, 2, 4, dtype=torch.float64, device=dev, generator=gen)
    shape = [lon.numel(), z.numel(), r.numel()]
    shape = [shape[i] for i in order]
    out = torch.randn([batch] + shape, dtype=torch.float64, device=dev, generator=gen)
    out *= 0.01
    s = torch.sqrt(1.0 - z * z)
    x = torch.cos(lon)[:, None, None] * s[None, :, None] * r[None, None, :]
    y = torch.sin(lon)[:, None, None] * s[None, :, None] * r[None, None, :]
    zz = (z[None, :, None] * r[None, None, :])
    r2 = (r * r)[None, None, :]
    for b in range(batch):
        for j in range(2):
            px, py, pz = (1.6 * c[b, j, k] - 0.8 for k in range(3))
            # |p - q|^2 = |p|^2 + |q|^2 - 2 p.q
            q = (r2 + (px * px + py * py + pz * pz)) - 2.0 * (px * x + py * y + pz * zz)
            out[b] += torch.exp(q * (-1.0 / (0.05 + 0.3 * c[b, j, 3]))).permute(order)
    return out.reshape(-1)


def _zt_grids(L, batch, gen):
    nlon, nlat, nrad = zg.zt_grid_shape(L)
    z, _ = _gl(nlat)
    x, _ = _gl(nrad)
    return _blobs(2.0 * np.pi * np.arange(nlon) / nlon, z, 0.5 * (1.0 + x), batch, gen, (0, 1, 2))


def _st_grids(L, latlon, batch, gen):
    a, b = zg.st_grid_shape(L, int(latlon))
    nlon, nlat = (b, a) if latlon else (a, b)
    z, _ = _gl(nlat)
    return _blobs(2.0 * np.pi * np.arange(nlon) / nlon, z, np.ones(1), batch, gen, (1, 0, 2) if latlon else (0, 1, 2))


def _euler(n, gen):
    """Rotations drawn uniformly."""
    u = torch.rand(n, 3, dtype=torch.float64, device=_device(), generator=gen)
    return torch.stack([2 * math.pi * u[:, 0], torch.acos(2 * u[:, 1] - 1), 2 * math.pi * u[:, 2]], 1).reshape(-1)


def _points(case, seed):
    """Points of an evaluation (lon, colat, rad) or of a fit, on the host as the callers hold them."""
    rng = np.random.default_rng(11 + seed)
    if case["op"] == "evaluate":
        return (rng.uniform(0, 2 * np.pi, case["nlon"]), np.arccos(rng.uniform(-1, 1, case["nlat"])),
                np.cbrt(rng.uniform(0, 1, case["nrad"])))
    n = case["points"]
    lon, z = rng.uniform(0, 2 * np.pi, n), rng.uniform(-1, 1, n)
    if case["kind"] == "st":
        return np.arcsin(z), lon  # latitudes, longitudes
    return np.cbrt(rng.uniform(0, 1, n)), lon, np.arccos(z)


def _inputs(case, seed):
    """The input tensors of a case, from the seed alone."""
    gen = _generator(seed)
    op, dev = case["op"], _device()
    new = lambda n: torch.zeros(n, dtype=torch.float64, device=dev)  # noqa: E731
    s = {}
    if op == "zt":
        L, Le, B = case["order"], case["exp_order"], case["batch"]
        csz, gsz = 2 * zg.zt_coeff_size(Le) * B, int(np.prod(zg.zt_grid_shape(L))) * B
        if case["mode"] == "backward":
            s["coeffs"] = _coefficients(_zt_scale(Le), B, gen)
        else:
            s["grids"] = _zt_grids(L, B, gen)
            s["coeffs"] = new(csz)
        if case["mode"] != "forward":
            s["out"] = new(gsz)
        if case["mode"] == "vjp":
            s["cot"] = _coefficients(_zt_scale(Le), B, gen)
    elif op == "st":
        L, Le, B, ll = case["order"], case["exp_order"], case["batch"], int(case["latlon"])
        csz, gsz = 2 * zg.st_coeff_size(Le) * B, int(np.prod(zg.st_grid_shape(L, ll))) * B
        if case["mode"] == "backward":
            s["coeffs"] = _coefficients(_st_scale(Le), B, gen)
        else:
            s["grids"] = _st_grids(L, ll, B, gen)
            s["coeffs"] = new(csz)
        if case["mode"] != "forward":
            s["out"] = new(gsz)
        if case["mode"] == "vjp":
            s["cot"] = _coefficients(_st_scale(Le), B, gen)
    elif op == "rotate":
        L, B = case["order"], case["batch"]
        scale = _zt_scale(L) if case["kind"] == "zt" else _st_scale(L)
        s["coeffs"] = _coefficients(scale, B, gen)
        s["euler"] = _euler(B, gen)
        s["work"] = new(scale.numel() * B)
        if case["grad"]:
            s["cot"] = _coefficients(scale, B, gen)
    elif op == "ragged":
        orders = _orders(case)
        scales = {int(L): _zt_scale(int(L)) for L in np.unique(orders)}
        s["orders"] = orders
        s["coeffs"] = torch.cat([_coefficients(scales[int(L)], int((orders == L).sum()), gen)
                                 for L in np.unique(orders)])
        s["euler"] = _euler(len(orders), gen)
        s["work"] = new(s["coeffs"].numel())
        s["out"] = new(int(sum(np.prod(zg.zt_grid_shape(int(L))) for L in orders)))
    elif op == "evaluate":
        L, B = case["order"], case["batch"]
        s["coeffs"] = _coefficients(_zt_scale(L) if case["kind"] == "zt" else _st_scale(L), B, gen)
        s["points"] = _points(case, seed)
        s["out"] = new(B * case["nlon"] * case["nlat"] * (case["nrad"] if case["kind"] == "zt" else 1))
    elif op == "lsq":
        s["points"] = tuple(torch.from_numpy(v).to(dev) for v in _points(case, seed))
        s["data"] = torch.randn(case["batch"] * case["points"], dtype=torch.float64, device=dev, generator=gen)
        size = zg.st_coeff_size(case["order"]) if case["kind"] == "st" else zg.zt_coeff_size(case["order"])
        s["out"] = new(2 * size * case["batch"])
    elif op == "spectra":
        L, B = case["order"], case["batch"]
        s["coeffs"] = _coefficients(_zt_scale(L) if case["kind"] == "zt" else _st_scale(L), B, gen)
        s["out"] = new(B * (L if case["kind"] == "st" else ((L + 1) * (L + 1)) >> 2))
    return s


def prepare(case, seed):
    state = _inputs(case, seed)
    state["case"], state["ctx"] = case, _context(case)
    return state


# ---- one pass ----------------------------------------------------------------------
def run(state):
    case, ctx, op = state["case"], state["ctx"], state["case"]["op"]
    if op in ("zt", "st"):
        L, Le, B, mode = case["order"], case["exp_order"], case["batch"], case["mode"]
        if op == "zt":
            conv, more = _zt_conv(case), {}
            forward, backward, vjp = ctx.zt_forward, ctx.zt_backward, ctx.zt_forward_vjp
        else:
            conv, more = _st_conv(case), {"layout": int(case["latlon"])}
            forward, backward, vjp = ctx.st_forward, ctx.st_backward, ctx.st_forward_vjp
        got = []
        if mode != "backward":
            got.append(forward(state["grids"], L, Le, B, conv, out=state["coeffs"], **more))
        if mode == "vjp":
            got.append(vjp(state["cot"], L, Le, B, conv, out=state["out"], **more))
        elif mode != "forward":
            got.append(backward(state["coeffs"], Le, L, B, conv, out=state["out"], **more))
        return got
    if op == "rotate":
        L, B, e, t = case["order"], case["batch"], state["euler"], case["type"]
        rotate, vjp = ((ctx.zt_rotate, ctx.zt_rotate_vjp) if case["kind"] == "zt" else
                       (ctx.st_rotate, ctx.st_rotate_vjp))
        state["work"].copy_(state["coeffs"])  # rotations are in place; the program keeps its expansions
        got = [rotate(state["work"], L, e, B, t)]
        if case["grad"]:
            got.extend(vjp(state["coeffs"], L, e, state["cot"], B, t))
        return got
    if op == "ragged":
        state["work"].copy_(state["coeffs"])
        ctx.zt_rotate_backward_ragged(state["orders"], state["work"], state["euler"], state["out"])
        return [state["work"], state["out"]]
    if op == "evaluate":
        lon, colat, rad = state["points"]
        if case["kind"] == "zt":
            return ctx.zt_evaluate(state["coeffs"], case["order"], lon, colat, rad, case["batch"], out=state["out"])
        return ctx.st_evaluate(state["coeffs"], case["order"], lon, colat, case["batch"], out=state["out"])
    if op == "lsq":
        fit = ctx.st_lsq if case["kind"] == "st" else ctx.zt_lsq
        return fit(state["data"], case["order"], *state["points"], batch=case["batch"], out=state["out"])
    power = ctx.st_power_spectrum if case["kind"] == "st" else ctx.zt_power_spectrum
    return power(state["coeffs"], case["order"], case["batch"], out=state["out"])


# ---- what a pass cannot do without ---------------------------------------------------
def _zt_transform_work(L, Le):
    """(bytes, flops) of one function, one direction: grid and coefficients once; an FFT of each (lat, rad)
    column, the Legendre sums folded over the equator and the radial sums."""
    Lm = min(L, Le)
    nlon, nlat, nrad = zg.zt_grid_shape(L)
    tri, zs = Lm * (Lm + 1) // 2, zg.zt_coeff_size(Lm)
    flops = 2.5 * nlon * math.log2(nlon) * nlat * nrad + 2.0 * tri * ((nlat + 1) // 2) * nrad * 2 + 4.0 * zs * nrad
    return 8.0 * nlon * nlat * nrad + 16.0 * zs, flops


def _st_transform_work(L, Le, latlon):
    Lm = min(L, Le)
    a, b = zg.st_grid_shape(L, int(latlon))
    nlon, nlat = (b, a) if latlon else (a, b)
    tri = Lm * (Lm + 1) // 2
    return 8.0 * nlon * nlat + 16.0 * tri, 2.5 * nlon * math.log2(nlon) * nlat + 4.0 * tri * ((nlat + 1) // 2)


def _rotate_work(kind, L):
    """(bytes, flops) of one rotation in place: the two X(+-pi/2) products, half of d(pi/2) each by parity."""
    if kind == "zt":
        n = [(L - l + 1) // 2 for l in range(L)]
    else:
        n = [1] * L
    flops = sum(c * 2 * 2.0 * (l + 1) * (l + 1) for l, c in enumerate(n))
    size = zg.zt_coeff_size(L) if kind == "zt" else zg.st_coeff_size(L)
    return 32.0 * size, flops


def work(case):
    op = case["op"]
    if op in ("zt", "st"):
        if op == "zt":
            by, fl = _zt_transform_work(case["order"], case["exp_order"])
        else:
            by, fl = _st_transform_work(case["order"], case["exp_order"], case["latlon"])
        f = case["batch"] * (2 if case["mode"] in ("round", "vjp") else 1)
        return {"bytes": by * f, "flops": fl * f}
    if op == "rotate":
        by, fl = _rotate_work(case["kind"], case["order"])
        # with the gradients: one more rotation, and five products in place of two
        f = case["batch"]
        return {"bytes": f * by * (3 if case["grad"] else 1), "flops": f * fl * (4.5 if case["grad"] else 1)}
    if op == "ragged":
        by = fl = 0.0
        for L in _orders(case):
            b0, f0 = _rotate_work("zt", int(L))
            b1, f1 = _zt_transform_work(int(L), int(L))
            by, fl = by + b0 + b1 - 16.0 * zg.zt_coeff_size(int(L)), fl + f0 + f1
        return {"bytes": by, "flops": fl}
    if op == "evaluate":
        L, B, nlon, nlat = case["order"], case["batch"], case["nlon"], case["nlat"]
        tri = L * (L + 1) // 2
        if case["kind"] == "zt":
            nrad = case["nrad"]
            zs = zg.zt_coeff_size(L)
            fl = 4.0 * zs * nrad + 4.0 * tri * nlat * nrad + 4.0 * L * nlon * nlat * nrad
            return {"bytes": B * (16.0 * zs + 8.0 * nlon * nlat * nrad), "flops": B * fl}
        return {"bytes": B * (16.0 * tri + 8.0 * nlon * nlat), "flops": B * (4.0 * tri * nlat + 4.0 * L * nlon * nlat)}
    if op == "lsq":
        L, m, B = case["order"], case["points"], case["batch"]
        n = L * L if case["kind"] == "st" else L * (L + 1) * (L + 2) // 6
        return {"bytes": 8.0 * m * (B + 3) + 8.0 * n * B,
                "flops": 2.0 * m * n * n - 2.0 / 3.0 * n ** 3 + 4.0 * m * n * B}
    L, B = case["order"], case["batch"]
    if case["kind"] == "st":
        return {"bytes": B * (16.0 * zg.st_coeff_size(L) + 8.0 * L), "flops": 4.0 * B * zg.st_coeff_size(L)}
    return {"bytes": B * (16.0 * zg.zt_coeff_size(L) + 2.0 * (L + 1) * (L + 1)), "flops": 4.0 * B * zg.zt_coeff_size(L)}


# ---- the same in 64 bits by torch and numpy alone --------------------------------------
def _plm(L, z, qm, cs):
    """P_lm(z) of the real basis, [l][m][z] (zero for m > l): normalised to 4 pi, or to 1 (qm)."""
    z = torch.as_tensor(z, dtype=torch.float64, device=_device())
    P = torch.zeros(L, L, z.numel(), dtype=torch.float64, device=z.device)
    u = torch.sqrt((1.0 - z) * (1.0 + z))
    d = torch.full_like(z, 1.0 if not qm else 1.0 / math.sqrt(4.0 * math.pi))
    for m in range(L):
        if m:
            d = d * u * math.sqrt((2.0 * m + 1.0) / (2.0 * m) * (2.0 if m == 1 else 1.0)) * (1.0 if cs else -1.0)
        P[m, m] = d
    m = torch.arange(L, dtype=torch.float64, device=z.device)[:, None]
    for l in range(1, L):
        k = m[:l]
        a = torch.sqrt((2.0 * l + 1.0) * (2.0 * l - 1.0) / ((l - k) * (l + k)))
        t = a * z * P[l - 1, :l]
        if l > 1:
            b = torch.sqrt((2.0 * l + 1.0) * (l + k - 1.0).clamp(min=0) * (l - k - 1.0).clamp(min=0) /
                           ((l - k) * (l + k) * (2.0 * l - 3.0)))
            t = t - b * P[l - 2, :l]
        P[l, :l] = t
    return P


def _radial(L, r, unnormed):
    """R_nl(r), [n][l][r]: r^l times the Jacobi polynomial P^(0, l + 1/2)_((n-l)/2)(2 r^2 - 1)."""
    r = torch.as_tensor(r, dtype=torch.float64, device=_device())
    R = torch.zeros(L, L, r.numel(), dtype=torch.float64, device=r.device)
    x = 2.0 * r * r - 1.0
    for l in range(L):
        b = l + 0.5
        p0, p1 = torch.ones_like(r), None
        for k in range((L - l + 1) // 2):
            if k == 0:
                p = p0
            elif k == 1:
                p = 1.0 + (b + 2.0) * 0.5 * (x - 1.0)
            else:
                c = 2.0 * k + b
                p = ((c - 1.0) * (c * (c - 2.0) * x - b * b) * p0 -
                     2.0 * (k - 1.0) * (k + b - 1.0) * c * p1) / (2.0 * k * (k + b) * (c - 2.0))
            if k:
                p0, p1 = p, p0
            n = l + 2 * k
            R[n, l] = p * r ** l * (1.0 if unnormed else math.sqrt(2.0 * n + 3.0))
    return R


class _Zt:
    """The Zernike transforms of one grid order as dense sums."""

    def __init__(self, L, Le, conv):
        self.L, self.Le, self.Lm = L, Le, min(L, Le)
        zn, qm, cs = conv
        self.unnormed, self.S = zn == 1, 1.0 if qm else 4.0 * math.pi
        self.nlon, self.nlat, self.nrad = zg.zt_grid_shape(L)
        z, self.wz = _gl(self.nlat)
        x, wr = _gl(self.nrad)
        r = 0.5 * (1.0 + x)
        dev = _device()
        self.w = torch.as_tensor(self.wz[:, None] * (0.5 * wr * r * r)[None, :], device=dev) * (2 * math.pi / self.nlon)
        self.P, self.R = _plm(self.Lm, z, qm, cs), _radial(self.Lm, r, self.unnormed)
        n, l, m = _zt_index(self.Lm)
        self.n, self.l, self.m = (torch.as_tensor(v, device=dev) for v in (n, l, m))

    def forward(self, g):
        X = torch.fft.rfft(g.reshape(self.nlon, self.nlat, self.nrad), dim=0)[:self.Lm]
        X = torch.stack([X.real, -X.imag], -1) * self.w[None, :, :, None]
        f = torch.einsum("lmj,mjkc->lmkc", self.P, X)
        c = torch.einsum("nlk,lmkc->nlmc", self.R, f)[self.n, self.l, self.m] / self.S
        if self.unnormed:
            c = c * (2.0 * self.n + 3.0)[:, None]
        out = torch.zeros(zg.zt_coeff_size(self.Le), 2, dtype=torch.float64, device=c.device)
        out[:c.shape[0]] = c
        return out.reshape(-1)

    def backward(self, c):
        d = torch.zeros(self.Lm, self.Lm, self.Lm, 2, dtype=torch.float64, device=c.device)
        d[self.n, self.l, self.m] = c.reshape(-1, 2)[:self.n.numel()]
        f = torch.einsum("nlk,nlmc->lmkc", self.R, d)
        X = torch.einsum("lmj,lmkc->mjkc", self.P, f) * (0.5 * self.nlon)
        X[0] *= 2.0
        F = torch.zeros(self.nlon // 2 + 1, self.nlat, self.nrad, dtype=torch.complex128, device=c.device)
        F[:self.Lm] = torch.complex(X[..., 0], -X[..., 1])
        return torch.fft.irfft(F, n=self.nlon, dim=0).reshape(-1)

    def adjoint(self, c):
        c = c.reshape(-1, 2)[:self.n.numel()] / self.S
        if self.unnormed:
            c = c * (2.0 * self.n + 3.0)[:, None]
        g = self.backward(torch.stack([c[:, 0], torch.where(self.m > 0, c[:, 1], 0.0)], 1).reshape(-1))
        return (g.reshape(self.nlon, self.nlat, self.nrad) * self.w).reshape(-1)


class _St:
    """The SH transforms of one grid order as dense sums."""

    def __init__(self, L, Le, conv, latlon):
        self.L, self.Le, self.Lm, self.latlon = L, Le, min(L, Le), latlon
        qm, cs = conv
        self.S = 1.0 if qm else 4.0 * math.pi
        a, b = zg.st_grid_shape(L, int(latlon))
        self.nlon, self.nlat = (b, a) if latlon else (a, b)
        z, w = _gl(self.nlat)
        w = w.copy()
        if latlon and self.nlat & 1:
            w[self.nlat // 2] *= 2.0  # the reference's fold counts the middle latitude of an odd grid twice
        self.w = torch.as_tensor(w, device=_device()) * (2 * math.pi / self.nlon)
        self.P = _plm(self.Lm, z, qm, cs)
        self.l, self.m = (torch.as_tensor(v, device=_device()) for v in _st_index(self.Lm))

    def forward(self, g):
        g = g.reshape(self.nlat, self.nlon).T if self.latlon else g.reshape(self.nlon, self.nlat)
        X = torch.fft.rfft(g, dim=0)[:self.Lm]
        X = torch.stack([X.real, -X.imag], -1) * self.w[None, :, None]
        c = torch.einsum("lmj,mjc->lmc", self.P, X)[self.l, self.m] / self.S
        out = torch.zeros(zg.st_coeff_size(self.Le), 2, dtype=torch.float64, device=c.device)
        out[:c.shape[0]] = c
        return out.reshape(-1)

    def backward(self, c):
        d = torch.zeros(self.Lm, self.Lm, 2, dtype=torch.float64, device=c.device)
        d[self.l, self.m] = c.reshape(-1, 2)[:self.l.numel()]
        X = torch.einsum("lmj,lmc->mjc", self.P, d) * (0.5 * self.nlon)
        X[0] *= 2.0
        F = torch.zeros(self.nlon // 2 + 1, self.nlat, dtype=torch.complex128, device=c.device)
        F[:self.Lm] = torch.complex(X[..., 0], -X[..., 1])
        g = torch.fft.irfft(F, n=self.nlon, dim=0)
        return (g.T if self.latlon else g).reshape(-1)

    def adjoint(self, c):
        c = c.reshape(-1, 2)[:self.l.numel()] / self.S
        g = self.backward(torch.stack([c[:, 0], torch.where(self.m > 0, c[:, 1], 0.0)], 1).reshape(-1))
        g = g.reshape(self.nlat, self.nlon) if self.latlon else g.reshape(self.nlon, self.nlat)
        return (g * (self.w[:, None] if self.latlon else self.w[None, :])).reshape(-1)


def _jy(l):
    """Eigenvectors of J_y of degree l (m = -l..l); its eigenvalues are -l..l in ascending order."""
    m = np.arange(-l, l)
    c = 0.5 * np.sqrt(l * (l + 1.0) - m * (m + 1.0))
    J = np.zeros((2 * l + 1, 2 * l + 1), dtype=np.complex128)
    J[m + 1 + l, m + l] = -1j * c
    J[m + l, m + 1 + l] = 1j * c
    return torch.from_numpy(np.linalg.eigh(J)[1]).to(_device())


def _rotated(c, euler, kind, L, rtype, jy):
    """Real expansions c [b][pairs][2] rotated by euler [b][3] (differentiable in both)."""
    if rtype == 0:
        al, be, ga = euler[:, 0], euler[:, 1], euler[:, 2]
    else:
        al, be, ga = -euler[:, 2], -euler[:, 1], -euler[:, 0]
    first = (lambda n, l: (n + 1) * (n + 3) * (2 * n + 1) // 24 + (l * l) // 4) if kind == "zt" else \
        (lambda n, l: l * (l + 1) // 2)
    rows, vals = [], []
    for l in range(L):
        at = [first(n, l) for n in (range(l, L, 2) if kind == "zt" else [l])]
        idx = torch.as_tensor(at, device=c.device)[:, None] + torch.arange(l + 1, device=c.device)[None, :]
        v = c[:, idx]  # b, vectors, m, 2
        m = torch.arange(l + 1, device=c.device)
        half = torch.full((l + 1,), math.sqrt(0.5), dtype=torch.float64, device=c.device)
        half[0] = 1.0
        pos = torch.complex(v[..., 0] * half, torch.where(m > 0, -v[..., 1] * half, 0.0 * v[..., 1]))
        sign = 1.0 - 2.0 * (m[1:] % 2)
        full = torch.cat([(pos[..., 1:].conj() * sign).flip(-1), pos], -1)
        k = torch.arange(-l, l + 1, dtype=torch.float64, device=c.device)
        phase = lambda t: torch.exp(-1j * t[:, None, None] * k)  # noqa: E731
        if l not in jy:
            jy[l] = _jy(l)
        V = jy[l]
        y = ((full * phase(ga)) @ V.conj()) * phase(be)
        y = ((y @ V.T) * phase(al))[..., l:]
        out = torch.stack([y.real / half, torch.where(m > 0, -y.imag / half, 0.0 * y.imag)], -1)
        rows.append(idx.reshape(-1))
        vals.append(out.reshape(c.shape[0], -1, 2))
    order = torch.argsort(torch.cat(rows))
    return torch.cat(vals, 1)[:, order]


def exact(case, seed):
    op, s = case["op"], _inputs(case, seed)
    if op in ("zt", "st"):
        B, mode = case["batch"], case["mode"]
        if op == "zt":
            t = _Zt(case["order"], case["exp_order"], _zt_conv(case))
        else:
            t = _St(case["order"], case["exp_order"], _st_conv(case), case["latlon"])
        each = lambda f, x: torch.cat([f(v) for v in x.reshape(B, -1)])  # noqa: E731
        if mode == "backward":
            return [each(t.backward, s["coeffs"])]
        c = each(t.forward, s["grids"])
        if mode == "forward":
            return [c]
        return [c, each(t.adjoint, s["cot"]) if mode == "vjp" else each(t.backward, c)]
    if op == "rotate":
        L, B, kind = case["order"], case["batch"], case["kind"]
        c, e, jy = s["coeffs"].reshape(B, -1, 2), s["euler"].reshape(B, 3), {}
        with torch.no_grad():
            got = [_rotated(c, e, kind, L, case["type"], jy).reshape(-1)]
        if case["grad"]:
            c.requires_grad_(True)
            e.requires_grad_(True)
            loss = (_rotated(c, e, kind, L, case["type"], jy).reshape(-1) * s["cot"]).sum()
            got.extend(g.reshape(-1) for g in torch.autograd.grad(loss, (c, e)))
        return got
    if op == "ragged":
        orders, jy, co, ro, cs, gs = s["orders"], {}, 0, 0, [], []
        for L in np.unique(orders):
            L, n = int(L), int((orders == L).sum())
            size = 2 * zg.zt_coeff_size(L)
            c = _rotated(s["coeffs"][co:co + n * size].reshape(n, -1, 2), s["euler"][3 * ro:3 * (ro + n)].reshape(n, 3),
                         "zt", L, 0, jy).reshape(n, -1)
            t = _Zt(L, L, (1, 0, 0) if zg.ZT_GEO[0] else (0, 0, 0))
            cs.append(c.reshape(-1))
            gs.extend(t.backward(v) for v in c)
            co, ro = co + n * size, ro + n
        return [torch.cat(cs), torch.cat(gs)]
    if op == "evaluate":
        L, B, pts = case["order"], case["batch"], _points(case, seed)
        P = _plm(L, np.cos(pts[1]), False, False)
        a = torch.as_tensor(pts[0], device=_device())[None, :] * torch.arange(L, device=_device())[:, None]
        trig = torch.stack([torch.cos(a), torch.sin(a)], -1)  # m, lon, c
        if case["kind"] == "zt":
            R = _radial(L, pts[2], zg.ZT_GEO[0] == 1)
            n, l, m = (torch.as_tensor(v, device=_device()) for v in _zt_index(L))
        else:
            l, m = (torch.as_tensor(v, device=_device()) for v in _st_index(L))
        out = []
        for c in s["coeffs"].reshape(B, -1, 2):
            if case["kind"] == "zt":
                d = torch.zeros(L, L, L, 2, dtype=torch.float64, device=c.device)
                d[n, l, m] = c
                f = torch.einsum("nlk,nlmc->lmkc", R, d)
            else:
                f = torch.zeros(L, L, 1, 2, dtype=torch.float64, device=c.device)
                f[l, m, 0] = c
            X = torch.einsum("lmj,lmkc->mjkc", P, f)
            out.append(torch.einsum("mic,mjkc->ijk", trig, X).reshape(-1))
        return torch.cat(out)
    if op == "lsq":
        L, B, pts = case["order"], case["batch"], s["points"]
        z = torch.sin(pts[0]) if case["kind"] == "st" else torch.cos(pts[2])
        P, lon = _plm(L, z, False, False), pts[1]
        if case["kind"] == "zt":
            R = _radial(L, pts[0], zg.ZT_GEO[0] == 1)
            idx = list(zip(*_zt_index(L)))
        else:
            idx = [(0, l, m) for l, m in zip(*_st_index(L))]
        cols, at = [], []
        for k, (n, l, m) in enumerate(idx):
            p = P[l, m] * R[n, l] if case["kind"] == "zt" else P[l, m]
            for c in range(2 if m else 1):
                cols.append(p * (torch.sin(int(m) * lon) if c else torch.cos(int(m) * lon)))
                at.append(2 * k + c)
        A = torch.stack(cols, 1)
        Q, U = torch.linalg.qr(A)
        x = torch.linalg.solve_triangular(U, Q.T @ s["data"].reshape(B, -1).T, upper=True)
        out = torch.zeros(B, 2 * len(idx), dtype=torch.float64, device=A.device)
        out[:, torch.as_tensor(at, device=A.device)] = x.T
        return out.reshape(-1)
    if op == "spectra":
        L, B = case["order"], case["batch"]
        p = s["coeffs"].reshape(B, -1, 2).square().sum(-1) / (4.0 * math.pi)
        if case["kind"] == "st":
            l = torch.as_tensor(_st_index(L)[0], device=p.device)
            return torch.zeros(B, L, dtype=torch.float64, device=p.device).index_add_(1, l, p).reshape(-1)
        n, l, _ = _zt_index(L)
        keep = torch.as_tensor(l < n, device=p.device)  # the reference's sum leaves l = n out
        at = torch.as_tensor((n + 1) * (n + 1) // 4 + l // 2, device=p.device)
        size = ((L + 1) * (L + 1)) >> 2
        out = torch.zeros(B, size, dtype=torch.float64, device=p.device)
        return out.index_add_(1, at[keep], p[:, keep]).reshape(-1)
    return None
