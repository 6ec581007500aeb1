"""Timed cases of the library's main path: treecode solves through the public entry points.

A case is a dict of plain values:

* ``kind``       "potential" (M free targets) or "force" (MRAG blocks of ``bs`` x ``bs`` targets)
* ``entry``      "device" (arrays resident in GPU memory, a caller's own ``Context``), "host"
                 (``Context.*_host`` on page-locked arrays), "plain" (the reference-compatible
                 ``treecode_*`` call on ordinary arrays) or "server" (a burst of requests)
* ``precision``  0 = plain FP64, 1 = mixed
* ``dist``       source distribution, as in ``workloads.py``: uniform, mixture, lamb, sheet
* ``n``, ``m``   sources, and targets (potential); ``g`` blocks per side (force)
* ``theta``      opening criterion; ``order``, ``bs``: expansion order and block side

``exact`` is the direct sum over all source-target pairs in 64 bits.
"""
import importlib
import math

import numpy as np
import torch

T = importlib.import_module("2d-treecodes_b200.treecodes")

EPS = 10 * 2.220446049250313e-16   # the softening of every pair, 10 DBL_EPSILON
EXACT_PAIRS = 2.5e11               # a direct sum of more pairs takes over about 20 seconds
CHUNK = 1 << 23                    # pairs of a direct sum held at once


def _case(name, kind, entry, precision, dist, n, m=0, g=0, theta=0.5, order=0, bs=32, requests=0):
    return dict(name=name, kind=kind, entry=entry, precision=precision, dist=dist, n=n, m=m, g=g,
                theta=theta, order=order or (12 if kind == "potential" else 24), bs=bs,
                requests=requests)


def listed():
    return [
        # the smallest request of a serving stream: 4K sources, one MRAG block; every step of a
        # small flow simulation pays this latency
        _case("force_4k", "force", "device", 1, "lamb", 4096, g=1),
        # the smallest potential: 4K sources and as many targets, all in FP64
        _case("potential_4k", "potential", "device", 0, "uniform", 4096, m=4096),
        # uniform sources with the targets at the sources, the ordinary small potential
        _case("potential_64k", "potential", "device", 0, "uniform", 65536, m=65536),
        # an odd number of sources, another number of targets, the tightest theta, mixed form
        _case("potential_ragged_mixed", "potential", "device", 1, "mixture", 700001, m=350003,
              theta=0.3),
        # clustered sources, as many targets, FP64: the largest potential
        _case("potential_4m", "potential", "device", 0, "mixture", 1 << 22, m=1 << 22),
        # a vortex with 32 x 32 blocks of 32 x 32 points in FP64: an ordinary flow step
        _case("force_1m", "force", "device", 0, "lamb", 1 << 20, g=32),
        # odd sizes, a lower order and smaller blocks, a loose theta, mixed form
        _case("force_ragged_order16", "force", "device", 1, "mixture", 300007, g=37, theta=0.7,
              order=16, bs=16),
        # a vortex sheet of 16M sources on 64 x 64 blocks, in both forms: the largest force
        _case("force_16m_mixed", "force", "device", 1, "sheet", 1 << 24, g=64),
        _case("force_16m", "force", "device", 0, "sheet", 1 << 24, g=64),
        # arrays in host memory: page-locked through a context, as a solver that overlaps does
        _case("force_host_1m", "force", "host", 0, "sheet", 1 << 20, g=32),
        # ordinary host arrays through the reference's own entry point
        _case("potential_host_131k", "potential", "plain", 0, "mixture", 131071, m=131071),
        # a burst of 12 requests of 4K to 256K sources to a request server with four slots
        _case("server_burst", "force", "server", 1, "lamb", 1 << 18, g=11, requests=12),
    ]


def draw(rng):
    kind = rng.choice(["potential", "force"])
    entry = rng.choice(["device"] * 6 + ["host", "plain"])
    precision = 0 if entry == "plain" else rng.choice([0, 1])
    theta = rng.choice([0.3, 0.5, 0.7])
    dist = rng.choice(["uniform", "mixture", "lamb", "sheet"])
    top = (1 << 20 if theta < 0.5 else 1 << 21) if kind == "potential" else 1 << 23
    if entry != "device":
        top = min(top, 1 << 20)
    n = int(round(math.exp(rng.uniform(math.log(4096), math.log(top)))))
    if rng.random() < 0.5:
        n |= 1
    order, bs, m, g = 0, 32, 0, 0
    if kind == "potential":
        m = n if rng.random() < 0.5 else max(1000, int(n * rng.uniform(0.2, 1.0)))
        if entry != "plain" and rng.random() < 0.25:
            order = rng.choice([8, 16, 20])
    else:
        if entry != "plain" and rng.random() < 0.25:
            order, bs = rng.choice([12, 16, 20]), rng.choice([16, 64])
        # about half as many targets as sources, as MRAG grids have
        g = max(1, round(math.sqrt(n * rng.uniform(0.25, 1.0)) / bs))
    c = _case("", kind, entry, precision, dist, n, m, g, theta, order, bs)
    del c["name"]
    return c


# ------------------------------------------------------------------------------- inputs
def _points(dist, n, gen):
    """Source coordinates and values of a distribution of workloads.py, drawn on the GPU."""
    def u(*s):
        return torch.rand(*s, generator=gen, device="cuda", dtype=torch.float64)

    def nrm(k):
        return torch.randn(k, generator=gen, device="cuda", dtype=torch.float64)

    if dist == "uniform":
        return u(n), u(n), 2 * u(n) - 1
    if dist == "mixture":
        centres = 0.1 + 0.8 * u(16, 2)
        sig = torch.exp(math.log(0.005) + math.log(10.0) * u(16))
        comp = torch.randint(0, 16, (n,), generator=gen, device="cuda")
        wide = u(n) < 0.2
        x = torch.where(wide, u(n), centres[comp, 0] + sig[comp] * nrm(n))
        y = torch.where(wide, u(n), centres[comp, 1] + sig[comp] * nrm(n))
        top = 1.0 - 2.0 ** -53
        return x.clamp(0.0, top), y.clamp(0.0, top), 2 * u(n) - 1
    if dist == "lamb":
        rad = 0.1 * torch.sqrt(-2 * torch.log1p(-u(n)))
        ang = 2 * math.pi * u(n)
        v = torch.exp(-rad * rad / 0.01) / n * (1 + 0.01 * nrm(n))
        return 0.5 + rad * torch.cos(ang), 0.5 + rad * torch.sin(ang), v
    x = u(n)
    y = 0.5 + 0.05 * torch.sin(2 * math.pi * x) + 0.002 * nrm(n)
    return x, y, (0.5 + u(n)) / n


def _grid(g, bs):
    """Origins and spacing of g x g blocks of bs x bs points over the unit square."""
    q = torch.arange(g * g, device="cuda", dtype=torch.float64)
    by = torch.floor(q / g)
    bx = q - g * by
    h = torch.full((g * g,), 1.0 / (g * bs), device="cuda", dtype=torch.float64)
    return bx / g, by / g, h


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = list(_points(case["dist"], case["n"], gen))
    if case["kind"] == "force":
        return s + list(_grid(case["g"], case["bs"]))
    if case["m"] == case["n"]:   # the targets at the sources
        return s + [s[0].clone(), s[1].clone()]
    t = _points(case["dist"], case["m"], gen)
    return s + [t[0], t[1]]


def _requests(case, seed):
    """A burst: kinds, distributions, thetas and sizes as a serving stream draws them."""
    r, out = np.random.Generator(np.random.PCG64(seed)), []
    for q in range(case["requests"]):
        n = int(round(math.exp(math.log(4096) + (q / (case["requests"] - 1)) *
                               math.log(case["n"] / 4096))))
        kind = "potential" if q % 3 == 2 else "force"
        out.append(dict(kind=kind, dist=("uniform", "mixture", "lamb", "sheet")[q % 4], n=n, m=n,
                        g=max(1, round(math.sqrt(n / 2048))), bs=32,
                        theta=(0.5, 0.7, 0.3)[(q // 2) % 3], seed=int(r.integers(1 << 30))))
    return out


def _host(t, pinned):
    if not pinned:
        return t.cpu().numpy()
    p = torch.empty(t.numel(), dtype=torch.float64, pin_memory=True)
    p.copy_(t)
    return p.numpy()


class _Burst:
    """A request server and the host arrays of a burst's requests."""

    def __init__(self, case, seed):
        self.server = T.Server(slots=4, hbm_budget_bytes=4 << 30)
        self.todo = [(q, [_host(t, True) for t in _inputs(q, q["seed"])])
                     for q in _requests(case, seed)]


def prepare(case, seed):
    if case["entry"] == "server":
        return dict(case=case, burst=_Burst(case, seed))
    a = _inputs(case, seed)
    state = dict(case=case)
    if case["entry"] != "plain":
        ctx = T.Context(precision=case["precision"])
        if case["kind"] == "potential":
            ctx.set_orders(potential_order=case["order"])
        else:
            ctx.set_orders(force_order=case["order"])
            ctx.set_blocksize(case["bs"])
        state["ctx"] = ctx
    nt = case["m"] if case["kind"] == "potential" else (case["g"] * case["bs"]) ** 2
    nout = 1 if case["kind"] == "potential" else 2
    if case["entry"] == "device":
        out = [torch.empty(nt, device="cuda", dtype=torch.float64) for _ in range(nout)]
    else:
        a = [_host(t, case["entry"] == "host") for t in a]
        out = [torch.empty(nt, dtype=torch.float64, pin_memory=True).numpy()
               for _ in range(nout)] if case["entry"] == "host" else []
    state.update(args=a, out=out)
    torch.cuda.synchronize()   # the library works on a stream of its own
    return state


def run(state):
    case = state["case"]
    potential = case["kind"] == "potential"
    if case["entry"] == "server":
        b, tickets = state["burst"], []
        for q, a in b.todo:
            submit = b.server.submit_potential if q["kind"] == "potential" else b.server.submit_force
            tickets.append(submit(q["theta"], *a, precision=case["precision"]))
        return [list(b.server.wait(t)[0]) for t in tickets]
    a, out, theta = state["args"], state["out"], case["theta"]
    if case["entry"] == "plain":
        call = T.treecode_potential if potential else T.treecode_force_mrag
        return call(theta, *a)
    ctx = state["ctx"]
    if case["entry"] == "host":
        call = ctx.potential_host if potential else ctx.force_mrag_host
    else:
        call = ctx.potential_device if potential else ctx.force_mrag_device
    return call(theta, *a, *out)


def _one_work(kind, n, nt, nb, order, theta):
    """Inputs read once, outputs written once; and the operations of one solve, modelled: the
    leaves' expansions and their merge; per target (force: per 8 x 8 brick of targets, plus one
    local series per target) the cells at a level that the opening criterion keeps, at every
    level, and the sources of the leaves around it."""
    force = kind == "force"
    leaf = 192 if force else 512
    levels = max(1.0, math.log(max(n / leaf, 1.0)) / math.log(4.0))
    disc = math.pi / (2 * theta * theta)   # area of the discs r < theta d, in cells
    cells = 3.0 * disc * levels
    near = min(float(n), disc * leaf / 2)
    up = n * 10 * order + n / leaf * 4 / 3 * (2 * order * order + 16 * order)
    if force:
        ev = nt * (10 * order + 11 * near) + nt / 64 * cells * (4 * order * order + 20 * order)
        return 24 * n + 24 * nb + 16 * nt, up + ev
    return 24 * n + 24 * nt, up + nt * (cells * (10 * order + 8) + 8 * near)


def work(case):
    if case["entry"] == "server":
        parts = [_one_work(q["kind"], q["n"], q["n"] if q["kind"] == "potential" else
                           (32 * q["g"]) ** 2, q["g"] ** 2,
                           12 if q["kind"] == "potential" else 24, q["theta"])
                 for q in _requests(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    nt = case["m"] if case["kind"] == "potential" else (case["g"] * case["bs"]) ** 2
    b, f = _one_work(case["kind"], case["n"], nt, case["g"] ** 2, case["order"], case["theta"])
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------- direct sums
def _direct(kind, a, bs):
    xs, ys, vs = a[:3]
    if kind == "force":
        x0, y0, h = a[3:]
        i = torch.arange(bs, device="cuda", dtype=torch.float64)
        shape = (len(x0), bs, bs)   # target (ix, iy) of block b at ix + bs (iy + bs b)
        xt = (x0[:, None, None] + h[:, None, None] * i[None, None, :]).expand(shape).reshape(-1)
        yt = (y0[:, None, None] + h[:, None, None] * i[None, :, None]).expand(shape).reshape(-1)
    else:
        xt, yt = a[3:]
    outs = [torch.empty_like(xt) for _ in range(2 if kind == "force" else 1)]
    step = max(1, CHUNK // len(xs))
    for k in range(0, len(xt), step):
        dx = xt[k:k + step, None] - xs
        dy = yt[k:k + step, None] - ys
        r2 = torch.addcmul(dx * dx, dy, dy).add_(EPS)
        if kind == "force":
            f = vs / r2
            outs[0][k:k + step] = dx.mul_(f).sum(1)
            outs[1][k:k + step] = dy.mul_(f).sum(1)
        else:
            outs[0][k:k + step] = r2.log_().mul_(vs).sum(1).mul_(0.5)
    return outs


def exact(case, seed):
    if case["entry"] == "server":
        out = []
        for q in _requests(case, seed):
            a = _inputs(q, q["seed"])
            out.append([o.cpu().numpy() for o in _direct(q["kind"], a, q["bs"])])
        return out
    nt = case["m"] if case["kind"] == "potential" else (case["g"] * case["bs"]) ** 2
    if float(case["n"]) * nt > EXACT_PAIRS:
        return None
    out = _direct(case["kind"], _inputs(case, seed), case["bs"])
    if case["entry"] != "device":
        out = [o.cpu().numpy() for o in out]
    return out[0] if case["kind"] == "potential" else tuple(out)
