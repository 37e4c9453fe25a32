"""The work whose speed counts: what a particle program has this framework do,
through its public entry points, from the smallest calls to the largest.

A case is one of eight kinds of call:

  step     a time step of a small simulation: new positions, update_positions,
           K * b (the operator follows the moved particles)
  count    new positions, update_positions, neighbour counts of every particle
  lists    host arrays in, host arrays out: a new particle set, its cell list,
           the neighbour lists of all particles
  sparse   K * b of a sparse (cut-off) operator
  dense    K * b of a dense operator
  fmm      K * b of a black-box FMM operator
  schwarz  the restricted additive Schwarz preconditioner: set-up and one apply
  solve    a whole RBF solve: learned preconditioner set-up and GMRES to 1e-8

Vectors and positions live on the GPU unless the kind says otherwise.  The
mixed-precision operators (FP32 pair terms) are called by programs that keep
their fields in single precision: their result is handed on as FP32.
"""
import math

import numpy as np
import torch

import aboria_gb300 as ab

MODELS = {2: "aboria_gb300/models/spai_mlp_2d.bin", 3: "aboria_gb300/models/spai_mlp_3d.bin"}
KINDS = {"gaussian": ab.K_GAUSSIAN, "wendland": ab.K_WENDLAND_C2, "laplace": ab.K_LAPLACE,
         "multiquadric": ab.K_MULTIQUADRIC, "compact_gaussian": ab.K_COMPACT_GAUSSIAN}
SOFTENING = 1e-3   # of the Laplace kernel, 1 / (|dx| + 1e-3)
MQ_C2 = 0.01       # of the multiquadric, sqrt(|dx|^2 + 0.1^2) (the reference's FMM test)
N_LEAF = 10.0      # particles per cell of the cell list (the reference's default)


def listed():
    return [
        # a small 2-D simulation: latency and launches are everything
        dict(name="step_2k", kind="step", n=2000, dim=2, points="uniform", periodic=True,
             neighbours=16.0, kernel="wendland", mixed=False),
        # the reference's CPU-runnable case as a moving particle set (50 neighbours each)
        dict(name="count_100k", kind="count", n=100_000, dim=3, points="uniform", periodic=False,
             radius=0.05),
        # neighbour counts of the benchmark's particle set: clustered, ~5,000 neighbours each
        dict(name="count_4m", kind="count", n=4_194_304, dim=3, points="mixture", periodic=True,
             radius=0.02),
        # neighbour lists for a program that works on the host
        dict(name="lists_50k", kind="lists", n=50_021, dim=3, points="uniform", periodic=True,
             radius=0.06),
        # the reference's CPU-runnable case: FP64 operator (the default precision)
        dict(name="sparse64_100k", kind="sparse", n=100_000, dim=3, points="uniform",
             periodic=False, radius=0.05, kernel="gaussian", mixed=False),
        # FP64 operator on a clustered set, ~1,200 neighbours each
        dict(name="sparse64_1m", kind="sparse", n=1_048_576, dim=3, points="mixture",
             periodic=True, radius=0.02, kernel="wendland", mixed=False),
        # the headline benchmark: mixed precision, 2.1e10 pairs
        dict(name="sparse32_4m", kind="sparse", n=4_194_304, dim=3, points="mixture",
             periodic=True, radius=0.02, kernel="wendland", mixed=True),
        # dense operator at its default precision, rows and columns different sets
        dict(name="dense64_32k", kind="dense", rows=32_768, cols=30_011, dim=3, kernel="gaussian",
             mixed=False),
        # FMM at its default order and precision
        dict(name="fmm64_1m_o3", kind="fmm", n=1_048_576, dim=3, order=3, kernel="laplace",
             mixed=False),
        # FMM at its highest benchmarked order, mixed precision
        dict(name="fmm32_1m_o7", kind="fmm", n=1_048_576, dim=3, order=7, kernel="laplace",
             mixed=True),
        # the reference's own preconditioner on an RBF system (leaves of 256 points)
        dict(name="schwarz_20k", kind="schwarz", n=20_000, dim=2, eps_h=2.5, leaf=256),
        # a whole RBF solve with the learned preconditioner
        dict(name="solve_200k", kind="solve", n=200_000, dim=2, eps_h=2.5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _ball(dim, r):
    return {1: 2.0 * r, 2: math.pi * r * r, 3: 4.0 / 3.0 * math.pi * r ** 3}[dim]


def _radius(n, dim, neighbours):
    """Radius of a ball that holds `neighbours` of n uniform points (at most a third of the box)."""
    return min((neighbours / n / _ball(dim, 1.0)) ** (1.0 / dim), 0.33)


def draw(rng):
    kind = rng.choice(["step", "count", "lists", "sparse", "sparse", "dense", "fmm", "fmm",
                       "schwarz", "solve"])
    dim = rng.choice([2, 3, 3])
    periodic = rng.random() < 0.5
    points = "mixture" if rng.random() < 0.4 else "uniform"
    if kind == "step":
        return dict(kind=kind, n=int(_log(rng, 500, 20_000)), dim=dim, points="uniform",
                    periodic=periodic, neighbours=rng.uniform(8.0, 60.0),
                    kernel=rng.choice(["gaussian", "wendland"]), mixed=rng.random() < 0.3)
    if kind in ("count", "lists", "sparse"):
        n = int(_log(rng, 2000, {"count": 2_000_000, "lists": 200_000, "sparse": 1_000_000}[kind]))
        # pairs stay below 2e8 (1e7 for the lists, which come back to the host)
        most = min(500.0, {"count": 2e8, "lists": 1e7, "sparse": 2e8}[kind] / n)
        if points == "mixture":
            most /= 8.0  # the clusters are denser than the mean
        r = _radius(n, dim, _log(rng, 6.0, max(most, 8.0)))
        c = dict(kind=kind, n=n, dim=dim, points=points, periodic=periodic, radius=r)
        if kind == "sparse":
            c["kernel"] = rng.choice(["gaussian", "wendland", "wendland", "compact_gaussian",
                                      "multiquadric", "laplace"])
            c["mixed"] = rng.random() < 0.4
        return c
    if kind == "dense":
        return dict(kind=kind, rows=int(_log(rng, 300, 32_768)), cols=int(_log(rng, 300, 32_768)),
                    dim=dim, kernel=rng.choice(["gaussian", "gaussian", "multiquadric", "laplace"]),
                    mixed=rng.random() < 0.4)
    if kind == "fmm":
        mixed = rng.random() < 0.5
        return dict(kind=kind, n=int(_log(rng, 5000, 1_000_000)), dim=dim,
                    order=rng.randint(3, 7 if mixed else 5),
                    kernel=rng.choice(["laplace", "laplace", "multiquadric"]), mixed=mixed)
    if kind == "schwarz":
        return dict(kind=kind, n=int(_log(rng, 2000, 20_000)), dim=2,
                    eps_h=rng.uniform(1.5, 3.0), leaf=rng.choice([64, 100, 256]))
    return dict(kind=kind, n=int(_log(rng, 5000, 200_000)), dim=dim, eps_h=rng.uniform(1.7, 3.0))


# ------------------------------------------------------------------ inputs ---
def _generator(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def _points(kind, n, dim, g):
    """n points of the unit box: uniform, or 16 Gaussian clusters (sigma 0.03)
    over a 20 % uniform background, wrapped into the box."""
    x = torch.rand(n, dim, generator=g, device="cuda", dtype=torch.float64)
    if kind == "uniform":
        return x
    centres = 0.1 + 0.8 * torch.rand(16, dim, generator=g, device="cuda", dtype=torch.float64)
    which = torch.randint(16, (n,), generator=g, device="cuda")
    spread = 0.03 * torch.randn(n, dim, generator=g, device="cuda", dtype=torch.float64)
    clustered = torch.rand(n, generator=g, device="cuda") < 0.8
    x = torch.where(clustered[:, None], (centres[which] + spread) % 1.0, x)
    return torch.where(x >= 1.0, torch.zeros_like(x), x)


def _turned(x, g):
    """The same configuration numbered, oriented and mirrored another way: the
    neighbour lists of two seeds differ and have the same length."""
    n, dim = x.shape
    x = x[torch.randperm(n, generator=g, device="cuda")]
    x = x[:, torch.randperm(dim, generator=g, device="cuda")]
    mirror = torch.rand(dim, generator=g, device="cuda") < 0.5
    x = torch.where(mirror, 1.0 - x, x)
    return torch.where(x >= 1.0, torch.zeros_like(x), x).contiguous()


def _normal(n, g):
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


def _case_radius(c):
    if "radius" in c:
        return c["radius"]
    if "eps_h" in c:
        return 4.0 / _eps(c)
    return _radius(c["n"], c["dim"], c["neighbours"])


def _eps(c):
    return c["eps_h"] * c["n"] ** (1.0 / c["dim"])


def _parameter(c):
    """The kernel's parameter p0."""
    k = c["kernel"]
    if k == "wendland":
        return 1.0 / _case_radius(c)
    if k in ("gaussian", "compact_gaussian"):
        # half the search radius for a cut-off operator, a broad one for a dense operator
        return 30.0 if c["kind"] == "dense" else 1.0 / (0.5 * _case_radius(c)) ** 2
    return SOFTENING if k == "laplace" else MQ_C2


def _kernel(c):
    return ab.Kernel.make(KINDS[c["kernel"]], _parameter(c))


def _precision(c):
    return ab.PREC_MIXED if c["mixed"] else ab.PREC_FP64


def _rhs(x):
    """Values to interpolate: a smooth field plus noise of 1e-3 from the points' own digits."""
    noise = torch.frac(x[:, 0] * 1e7) - 0.5
    return torch.sin(4 * math.pi * x[:, 0]) * torch.cos(3 * math.pi * x[:, 1]) + 1e-3 * noise


_shared = {}


def _stream():
    """The program's own stream, which the framework's context shares."""
    if not _shared:
        s = torch.cuda.Stream()
        _shared["stream"], _shared["ctx"] = s, ab.Context(0, stream=s.cuda_stream)
    return _shared["stream"]


def prepare(c, seed):
    stream = _stream()
    ctx = _shared["ctx"]
    with torch.cuda.stream(stream):
        g = _generator(seed)
        kind, dim = c["kind"], c.get("dim", 3)
        s = dict(c, case_kind=kind, ctx=ctx, lo=[0.0] * dim, hi=[1.0] * dim)
        box = (s["lo"], s["hi"], [c.get("periodic", False)] * dim)
        s["box"] = box
        if kind == "dense":
            rows = ab.Particles(dim, ctx).set(_points("uniform", c["rows"], dim, g))
            cols = ab.Particles(dim, ctx).set(_points("uniform", c["cols"], dim, g))
            s["K"] = ab.create_dense_operator(rows, cols, _kernel(c), _precision(c))
            s["b"] = _normal(c["cols"], g)
        else:
            if kind == "lists":
                x = _turned(_points(c["points"], c["n"], dim, _generator(c["n"])), g)
                s["x"], s["p"] = x.cpu().numpy(), ab.Particles(dim, ctx)
                s["r"] = _case_radius(c)
            else:
                x = _points(c.get("points", "uniform"), c["n"], dim, g)
                p = s["p"] = ab.Particles(dim, ctx).set(x)
                if kind in ("step", "count", "sparse"):
                    p.init_neighbour_search(*box, N_LEAF)
                    s["r"] = _case_radius(c)
                elif kind == "fmm":
                    p.init_octree(*box, 64)
                    s["K"] = ab.create_fmm_operator(p, _kernel(c), c["order"], _precision(c))
                else:
                    p.init_octree(*box, c.get("leaf", 256))
                    kern = ab.Kernel.make(ab.K_COMPACT_GAUSSIAN, _eps(c) ** 2)
                    s["K"] = ab.create_sparse_operator(p, p, _case_radius(c), kern, ab.PREC_FP64)
                    s["b"] = _rhs(x[torch.from_numpy(p.ids).cuda()])
                if kind in ("step", "sparse"):
                    s["K"] = ab.create_sparse_operator(p, p, s["r"], _kernel(c), _precision(c))
                if kind in ("step", "count"):
                    s["x"] = _points(c["points"], c["n"], dim, g)  # where the particles move to
                if kind in ("step", "sparse", "fmm"):
                    s["b"] = _normal(c["n"], g)
                if kind == "solve":
                    s["mlp"] = ab.MLP.load(MODELS[dim], ctx)
        torch.cuda.synchronize()
    return s


def run(s):
    kind = s["case_kind"]
    with torch.cuda.stream(_stream()):
        if kind in ("sparse", "dense", "fmm"):
            y = s["K"] * s["b"]
            return y.float() if s["mixed"] else y
        if kind == "step":
            s["p"].set_positions(s["x"])
            s["p"].update_positions()
            y = s["K"] * s["b"]
            return y.float() if s["mixed"] else y
        if kind == "count":
            s["p"].set_positions(s["x"])
            s["p"].update_positions()
            counts = torch.empty(s["n"], dtype=torch.int32, device="cuda")
            return ab.radius_count(s["p"], s["x"], s["r"], out=counts)
        if kind == "lists":
            s["p"].set(s["x"])
            s["p"].init_neighbour_search(*s["box"], N_LEAF)
            rowptr, cols = ab.radius_query_csr(s["p"], s["x"], s["r"])
            return rowptr, cols, s["p"].ids
        if kind == "schwarz":
            return ab.schwarz_preconditioner(s["K"]).solve(s["b"])
        M = ab.learned_preconditioner(s["K"], s["mlp"], _eps(s))
        x, _, _ = ab.gmres(s["K"], s["b"], M=M, restart=100, max_iters=300, tol=1e-8)
        return x


# -------------------------------------------------------------------- work ---
def _mean_neighbours(c):
    r, dim, n = _case_radius(c), c["dim"], c["n"]
    uniform = _ball(dim, r)
    if c.get("points", "uniform") == "uniform":
        return n * min(uniform, 1.0)
    # two points of one cluster lie within r with probability P(chi_dim < r / (sigma sqrt 2))
    a = r / (2.0 * 0.03)
    if dim == 3:
        p = math.erf(a) - 2.0 * a / math.sqrt(math.pi) * math.exp(-a * a)
    else:
        p = 1.0 - math.exp(-a * a) if dim == 2 else math.erf(a)
    return n * (0.64 / 16.0 * p + (1.0 - 0.64 / 16.0) * min(uniform, 1.0))


def work(c):
    kind, dim, n = c["kind"], c.get("dim", 3), c.get("n", 0)
    if kind == "dense":
        pairs = c["rows"] * c["cols"]
        return {"bytes": 8.0 * (dim * (c["rows"] + c["cols"]) + c["rows"] + c["cols"]),
                "flops": 11.0 * pairs}
    if kind == "fmm":
        nodes = c["order"] ** dim
        leaves = max(1.0, n / 32.0)
        m2l = leaves * (189.0 if dim == 3 else 27.0) * 2.0 * nodes * nodes
        near = n * 32.0 * 3.0 ** dim * 11.0
        return {"bytes": 8.0 * n * (dim + 2), "flops": m2l + near + 4.0 * n * nodes}
    pairs = n * max(_mean_neighbours(c), 1.0)
    if kind in ("count", "step"):
        move = n * (16.0 * dim + 24.0)
        return {"bytes": move + 16.0 * n, "flops": (8.0 if kind == "count" else 20.0) * pairs}
    if kind == "lists":
        return {"bytes": n * (16.0 * dim + 24.0) + 4.0 * pairs, "flops": 8.0 * pairs}
    if kind == "sparse":
        return {"bytes": 8.0 * n * (dim + 2), "flops": 20.0 * pairs}
    if kind == "schwarz":
        size = min(float(n), 9.0 * 0.6 * c["leaf"])
        domains = n / (0.6 * c["leaf"])
        return {"bytes": domains * 8.0 * size * size, "flops": domains * 2.0 / 3.0 * size ** 3}
    # solve: about ten matvecs, applies of 32 entries a row, and orthogonalisations
    infer = 2.0 * n * (32 * dim * 128 + 2 * 128 * 128 + 128 * 32)
    return {"bytes": 10.0 * n * (8.0 * (dim + 2) + 32 * 12.0 + 10 * 16.0),
            "flops": 10.0 * n * (20.0 * pairs / n + 64.0) + infer}


# ------------------------------------------------------------------- exact ---
def _kernel_value(k, d2, p0):
    if k == "wendland":
        q = (torch.sqrt(d2) * p0).clamp(max=1.0)
        return (1.0 - q) ** 4 * (4.0 * q + 1.0)
    if k in ("gaussian", "compact_gaussian"):
        return torch.exp(-d2 * p0)
    if k == "laplace":
        return 1.0 / (torch.sqrt(d2) + p0)
    return torch.sqrt(d2 + p0)


def _storage_order(x):
    """Order of the cell list: stable by cell, last dimension fastest."""
    n, dim = x.shape
    size = max(1, int(math.floor(1.0 / (N_LEAF / n) ** (1.0 / dim))))
    key = torch.zeros(n, dtype=torch.int64, device=x.device)
    for d in range(dim):
        key = key * size + torch.floor(x[:, d] * size).long().clamp(0, size - 1)
    return torch.argsort(key, stable=True)


def _octree_order(x):
    """Order of the octree: stable by the interleaved bits of the coordinates."""
    n, dim = x.shape
    levels = 32 // dim - 2
    cells = [torch.floor(x[:, d] * 2.0 ** levels).long() for d in range(dim)]
    key = torch.zeros(n, dtype=torch.int64, device=x.device)
    for bit in range(levels - 1, -1, -1):
        for d in range(dim):
            key = key * 2 + ((cells[d] >> bit) & 1)
    return torch.argsort(key, stable=True)


def _pair_chunks(rows, x, r, periodic, most=30_000_000):
    """All (row, column) pairs within r, with their squared distances, in
    chunks of rows: columns binned into cells of side >= r, periodic images
    added as points outside the box."""
    dim, dev = x.shape[1], x.device
    index = torch.arange(len(x), device=dev)
    pts = x
    if periodic:
        for d in range(dim):
            low, high = pts[:, d] <= r, pts[:, d] >= 1.0 - r
            shift = torch.zeros(dim, dtype=torch.float64, device=dev)
            shift[d] = 1.0
            pts, index = (torch.cat([pts, pts[low] + shift, pts[high] - shift]),
                          torch.cat([index, index[low], index[high]]))
    m = max(1, min(int(1.0 / r * (1.0 - 1e-9)), 200 if dim == 3 else 2000))
    w = m + 4  # two cells of margin on every side

    def cells(y):
        return [(torch.floor(y[:, d] * m).long() + 2).clamp(0, w - 1) for d in range(dim)]

    def join(c):
        key = torch.zeros_like(c[0])
        for d in range(dim):
            key = key * w + c[d]
        return key

    key, order = torch.sort(join(cells(pts)))
    pts, index = pts[order], index[order]
    start = torch.searchsorted(key, torch.arange(w ** dim + 1, device=dev))
    rc = cells(rows)
    offsets = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)] if dim == 3 else [(a,) for a in (-1, 0, 1)]
    first = torch.stack([start[join([rc[d] + o[d] for d in range(dim - 1)] + [rc[-1] - 1])] for o in offsets], 1)
    last = torch.stack([start[join([rc[d] + o[d] for d in range(dim - 1)] + [rc[-1] + 1]) + 1] for o in offsets], 1)
    total = torch.cumsum((last - first).sum(1), 0).cpu().numpy()
    at = 0
    while at < len(rows):
        base = total[at - 1] if at else 0
        to = max(at + 1, int(np.searchsorted(total, base + most, side="right")))
        length = (last[at:to] - first[at:to]).reshape(-1)
        row = torch.arange(at, to, device=dev).repeat_interleave(len(offsets)).repeat_interleave(length)
        skip = torch.cumsum(length, 0) - length
        col = torch.arange(len(row), device=dev) + (first[at:to].reshape(-1) - skip).repeat_interleave(length)
        d2 = torch.zeros(len(row), dtype=torch.float64, device=dev)
        for d in range(dim):
            d2 += (pts[col, d] - rows[row, d]) ** 2
        inside = d2 <= r * r
        yield row[inside], index[col[inside]], d2[inside]
        at = to


def _sparse_product(x, r, periodic, kernel, p0, b):
    c = torch.zeros(len(x), dtype=torch.float64, device=x.device)
    for row, col, d2 in _pair_chunks(x, x, r, periodic):
        c.index_add_(0, row, _kernel_value(kernel, d2, p0) * b[col])
    return c


def _dense_product(rows, cols, kernel, p0, b):
    out = []
    for part in rows.split(max(1, 30_000_000 // len(cols))):
        d2 = sum((part[:, None, d] - cols[None, :, d]) ** 2 for d in range(rows.shape[1]))
        out.append((_kernel_value(kernel, d2, p0) * b).sum(1))
    return torch.cat(out)


def _solve_exact(x, r, eps2, f):
    """The interpolation system by conjugate gradients in 64 bits, to rounding
    (the truncated Gaussian matrix of well separated scales is positive)."""
    n = len(x)
    parts = [(i, j, torch.exp(-eps2 * d2)) for i, j, d2 in _pair_chunks(x, x, r, False)]
    i, j, v = (torch.cat([p[k] for p in parts]) for k in range(3))
    A = torch.sparse_coo_tensor(torch.stack([i, j]), v, (n, n)).coalesce().to_sparse_csr()
    y = torch.zeros_like(f)
    res = f.clone()
    d = res.clone()
    rr = res @ res
    stop = 1e-28 * rr
    for _ in range(3000):
        if rr <= stop:
            break
        q = A @ d
        alpha = rr / (d @ q)
        y += alpha * d
        res -= alpha * q
        new = res @ res
        d = res + (new / rr) * d
        rr = new
    return y


def exact(c, seed):
    kind, dim, n = c["kind"], c.get("dim", 3), c.get("n", 0)
    if kind == "schwarz":
        return None  # sums over overlapping subdomain solves have no shorter formula
    g = _generator(seed)
    if kind == "dense":
        rows = _points("uniform", c["rows"], dim, g)
        cols = _points("uniform", c["cols"], dim, g)
        return _dense_product(rows, cols, c["kernel"], _parameter(c), _normal(c["cols"], g))
    x = _points(c.get("points", "uniform"), n, dim, g)
    if kind in ("count", "lists") or (kind == "fmm" and n > 60_000):
        return None  # whole numbers; a direct sum of more points takes too long
    if kind == "solve":
        x = x[_octree_order(x)]
        return _solve_exact(x, _case_radius(c), _eps(c) ** 2, _rhs(x))
    if kind == "fmm":
        x = x[_octree_order(x)]
        return _dense_product(x, x, c["kernel"], _parameter(c), _normal(n, g))
    if n * _mean_neighbours(c) > 3e9:
        return None
    if kind == "step":
        x = _points(c["points"], n, dim, g)
    x = x[_storage_order(x)]
    return _sparse_product(x, _case_radius(c), c["periodic"], c["kernel"], _parameter(c), _normal(n, g))
