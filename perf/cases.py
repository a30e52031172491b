"""The timed workloads of the KDTree path: what a user of the package has it do.

Every case is one pass through the public entry points (`KDTree`, `BatchedDensity`) on
synthetic particles of the kinds the benchmark and the tests use: uniform periodic boxes,
boxes with 70% of the particles in 500 Plummer spheres (the rest a uniform background), and
batches of separate groups with power-law sizes. Inputs are made on the device from the seed.

Passes whose particles are new each time (a snapshot, a group catalogue, an optimiser step)
include the tree build; passes that put several queries to one tree (ball search, smoothing,
field values at points) keep the tree, as such a program does.

`listed()` gives the named cases, `draw(rng)` others from the same ranges, `prepare` the
state of a case, `run` one pass and its outputs, `work` the bytes and operations a pass
cannot do without, `exact` the outputs in plain 64-bit torch where that is quick.
"""
from __future__ import annotations

import math

import torch

from nbodylib_gb300 import BatchedDensity, KDTree
from nbodylib_gb300.kdtree import FOF6D, KSPH, TPHS

DEV = "cuda"
BUCKET = 16
MINNUM = 20
KERNRES = 1000


def listed():
    return [
        # one halo candidate handed over from host arrays and linked: the smallest call of a
        # halo finder's inner loop, latency and launches only
        {"name": "fof_group_host", "kind": "fof", "n": 5003, "spheres": 8, "periodic": False,
         "host": True},
        # a simulation snapshot: tree build + friends-of-friends in a periodic box
        {"name": "fof_box", "kind": "fof", "n": 1 << 20, "spheres": 500, "periodic": True,
         "host": False},
        # a small periodic box: neighbour lists and densities of every particle
        {"name": "knn_uniform_box", "kind": "knn", "n": 32768, "k": 32, "uniform": True,
         "periodic": True},
        # the density of every particle of a snapshot (build, CalcDensity, delete)
        {"name": "density_box", "kind": "density", "n": 1 << 20, "k": 32},
        # a large snapshot: density and velocity density with k = 64 on one tree
        {"name": "veldensity_256cubed", "kind": "veldensity", "n": 256 ** 3, "k": 64},
        # a group catalogue: every group its own tree, built and searched together
        {"name": "batch_groups", "kind": "batch", "groups": 20000, "nmin": 20, "nmax": 200000,
         "k": 32},
        # one step of an optimisation through the density: build, forward and gradients
        {"name": "adjoint_box", "kind": "adjoint", "n": 1 << 20, "k": 32},
        # phase-space linking of a snapshot: build + FOFCriterion with FOF6d
        {"name": "fof6d_box", "kind": "fof6d", "n": 1 << 20},
        # phase-space density with the local metric (TreeType TPHS): build + CalcDensity
        {"name": "phase_density", "kind": "phase", "n": 1 << 18, "k": 32},
        # every particle's neighbours within a radius, on a kept tree
        {"name": "ball_box", "kind": "ball", "n": 1 << 20, "per_ball": 32.0},
        # smoothed velocity and velocity dispersion fields, on a kept tree with its density
        {"name": "smooth_box", "kind": "smooth", "n": 1 << 20, "k": 32},
        # field values at points that are not particles (a ragged number of sightline or grid
        # points): neighbour lists and densities at the points, on a kept tree
        {"name": "points_field", "kind": "points", "n": 500009, "points": 250007, "k": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    kind = rng.choice(["fof", "fof", "knn", "density", "veldensity", "batch", "adjoint", "fof6d",
                       "phase", "ball", "smooth", "points"])
    if kind == "fof":
        n = _log_int(rng, 1000, 4000000)
        return {"kind": kind, "n": n, "spheres": 8 if n < 50000 else 500,
                "periodic": rng.random() < 0.5, "host": n < 50000}
    if kind == "knn":
        return {"kind": kind, "n": _log_int(rng, 5000, 1000000), "k": rng.randint(8, 64),
                "uniform": rng.random() < 0.5, "periodic": rng.random() < 0.5}
    if kind == "density":
        return {"kind": kind, "n": _log_int(rng, 5000, 4000000), "k": rng.randint(8, 64)}
    if kind == "veldensity":
        return {"kind": kind, "n": _log_int(rng, 100000, 4000000), "k": rng.randint(16, 64)}
    if kind == "batch":
        return {"kind": kind, "groups": _log_int(rng, 50, 20000), "nmin": rng.randint(20, 40),
                "nmax": _log_int(rng, 2000, 200000), "k": rng.randint(16, 40)}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_int(rng, 20000, 1000000), "k": rng.randint(16, 64)}
    if kind == "fof6d":
        return {"kind": kind, "n": _log_int(rng, 20000, 1000000)}
    if kind == "phase":
        return {"kind": kind, "n": _log_int(rng, 10000, 300000), "k": rng.randint(16, 40)}
    if kind == "ball":
        return {"kind": kind, "n": _log_int(rng, 20000, 1500000),
                "per_ball": round(rng.uniform(8.0, 64.0), 2)}
    if kind == "smooth":
        return {"kind": kind, "n": _log_int(rng, 20000, 1000000), "k": rng.randint(16, 64)}
    return {"kind": kind, "n": _log_int(rng, 20000, 1000000),
            "points": _log_int(rng, 5000, 500000), "k": rng.randint(16, 64)}


# ---- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _box_side(n):
    """The benchmark's number density: 2^20 particles in a box of side 100."""
    return 100.0 * (n / float(1 << 20)) ** (1.0 / 3.0)


def _plummer(g, a):
    """Radii of Plummer spheres of scale a, inside 10 a."""
    u_max = (10.0 / math.sqrt(101.0)) ** 3  # the mass fraction inside 10 a
    u = _rand(g, a.numel()).clamp_min_(1e-12) * u_max
    r = a / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    d = _randn(g, a.numel(), 3)
    return r[:, None] * d / d.norm(dim=1, keepdim=True)


def _clustered(g, n, spheres=500, velocities=False):
    """70% of n particles in Plummer spheres (members dN/dn ~ n^-2, scale radii log-uniform
    in [0.05, 0.5]), the rest uniform, in the periodic box of side _box_side(n)."""
    box = _box_side(n)
    nc = int(round(0.7 * n))
    raw = 1.0 / (1.0 - _rand(g, spheres))
    edges = torch.floor(torch.cumsum(raw, 0) / raw.sum() * nc).to(torch.int64)
    edges[-1] = nc
    sphere = torch.searchsorted(edges, torch.arange(nc, device=DEV), right=True)
    centres = _rand(g, spheres, 3) * box
    scale = torch.exp(math.log(0.05) + _rand(g, spheres) * math.log(10.0))
    pos = torch.cat([centres[sphere] + _plummer(g, scale[sphere]), _rand(g, n - nc, 3) * box])
    pos = torch.remainder(pos, box)
    pos = torch.where(pos >= box, torch.zeros_like(pos), pos)
    vel = None
    if velocities:  # per sphere the Plummer dispersion, 0.1 for the background
        counts = torch.diff(edges, prepend=edges.new_zeros(1)).to(torch.float64)
        sig = torch.sqrt(3.0 * math.pi / 64.0 * (counts / n) / scale)
        vel = torch.cat([_randn(g, nc, 3) * sig[sphere][:, None], _randn(g, n - nc, 3) * 0.1])
    order = torch.randperm(n, generator=g, device=DEV)  # files are not sorted by object
    mass = (0.5 + _rand(g, n)) / n
    return pos[order].contiguous(), None if vel is None else vel[order].contiguous(), mass, box


def _groups(g, case):
    """Groups of Plummer spheres (a = 1) with dN/dn ~ n^-2 sizes on [nmin, nmax]."""
    lo, hi = 1.0 / case["nmin"], 1.0 / case["nmax"]
    # the sizes are those of the quantiles, so that the particles of a case hardly vary
    u = (torch.arange(case["groups"], device=DEV, dtype=torch.float64) + 0.5) / case["groups"]
    u = u[torch.randperm(case["groups"], generator=g, device=DEV)]
    sizes = torch.floor(1.0 / (lo - u * (lo - hi))).to(torch.int64)
    off = torch.zeros(case["groups"] + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(sizes, 0, out=off[1:])
    total = int(off[-1])
    pos = _plummer(g, torch.ones(total, device=DEV, dtype=torch.float64))
    return pos, 0.5 + _rand(g, total), off


def _inputs(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        pos, mass, off = _groups(g, case)
        return {"pos": pos, "mass": mass, "off": off}
    n = case["n"]
    if case.get("uniform") or kind == "ball":
        return {"pos": _rand(g, n, 3), "mass": (0.5 + _rand(g, n)) / n, "box": 1.0}
    pos, vel, mass, box = _clustered(g, n, case.get("spheres", 500),
                                     kind in ("veldensity", "fof6d", "phase", "smooth"))
    x = {"pos": pos, "mass": mass, "box": box}
    if vel is not None:
        x["vel"] = vel
    if kind == "adjoint":
        x["w"] = _randn(g, n)
    if kind == "points":  # two thirds near particles, the rest anywhere in the box
        m = case["points"]
        near = (2 * m) // 3
        at = torch.randint(n, (near,), generator=g, device=DEV)
        x["points"] = torch.cat([pos[at] + _randn(g, near, 3) * 0.05, _rand(g, m - near, 3) * box])
    return x


def _radius2(case):
    return (3.0 * case["per_ball"] / (4.0 * math.pi * case["n"])) ** (2.0 / 3.0)


def prepare(case, seed):
    x = _inputs(case, seed)
    s = {"case": dict(case), **x}
    kind = case["kind"]
    if case.get("host"):
        s["pos"], s["mass"] = x["pos"].cpu().numpy(), x["mass"].cpu().numpy()
    if kind == "ball":
        s["tree"] = KDTree(s["pos"], None, s["mass"], BUCKET, kerntype=KSPH, period=[1.0] * 3,
                           device=True)
        s["targets"] = torch.arange(case["n"], dtype=torch.int32, device=DEV)
        # the program's own list buffer, a tenth larger than the lists are expected to be
        s["lists"] = torch.full((int(1.1 * case["per_ball"] * case["n"]) + 4096,), -1,
                                dtype=torch.int32, device=DEV)
    elif kind == "smooth":
        s["tree"] = KDTree(s["pos"], s["vel"], s["mass"], BUCKET, kerntype=KSPH, device=True)
        s["rho"] = s["tree"].CalcDensity(case["k"])
    elif kind == "points":
        s["tree"] = KDTree(s["pos"], None, s["mass"], BUCKET, kerntype=KSPH,
                           period=[s["box"]] * 3, device=True)
    return s


# ---- one pass

def _linking_length(s):
    return 0.2 * s["box"] / s["case"]["n"] ** (1.0 / 3.0)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "fof":
        period = [s["box"]] * 3 if case["periodic"] else None
        t = KDTree(s["pos"], None, s["mass"], BUCKET, kerntype=KSPH, period=period,
                   device=not case["host"])
        group, ngroup = t.FOF(_linking_length(s), MINNUM)
        t.close()
        return group, ngroup
    if kind == "knn":
        period = [s["box"]] * 3 if case["periodic"] else None
        t = KDTree(s["pos"], None, s["mass"], BUCKET, kerntype=KSPH, period=period, device=True)
        nn, d2 = t.FindNearest(case["k"])
        perm = t.GetPerm()
        rho = t.CalcDensity(case["k"])
        t.close()
        return {"nn": nn, "d2": d2, "perm": perm, "rho": rho}
    if kind == "density":
        t = KDTree(s["pos"], None, s["mass"], BUCKET, kerntype=KSPH, device=True)
        rho = t.CalcDensity(case["k"])
        t.close()
        return rho
    if kind == "veldensity":
        t = KDTree(s["pos"], s["vel"], s["mass"], BUCKET, kerntype=KSPH, device=True)
        rho = t.CalcDensity(case["k"])
        vden = t.CalcVelDensity(case["k"], case["k"])
        t.close()
        return rho, vden
    if kind == "batch":
        b = BatchedDensity(s["pos"], s["mass"], s["off"], bucket_size=BUCKET, kerntype=KSPH,
                           device=True)
        b.set_stream(torch.cuda.current_stream())
        rho = b.density(case["k"], use_graph=False)
        b.close()
        return rho
    if kind == "adjoint":
        t = KDTree(s["pos"], None, s["mass"], BUCKET, kerntype=KSPH, device=True)
        rho, gpos, gmass = t.DensityAdjoint(case["k"], s["w"])
        t.close()
        return rho, gpos, gmass
    if kind == "fof6d":
        ll2 = _linking_length(s) ** 2
        t = KDTree(s["pos"], s["vel"], s["mass"], BUCKET, kerntype=KSPH, period=[s["box"]] * 3,
                   device=True)
        group, ngroup = t.FOFCriterion(FOF6D, [0, ll2, 0, 0, 0, 0, ll2, 0.04], MINNUM)
        t.close()
        return group, ngroup
    if kind == "phase":
        t = KDTree(s["pos"], s["vel"], s["mass"], BUCKET, treetype=TPHS, kerntype=KSPH,
                   device=True)
        rho = t.CalcDensity(case["k"])
        t.close()
        return rho
    if kind == "ball":
        offsets, found = s["tree"].SearchBallPosTagged(s["targets"], _radius2(case))
        s["lists"][:found.numel()].copy_(found)  # as handed on, with the offsets
        return offsets, s["lists"]
    if kind == "smooth":
        mean = s["tree"].CalcSmoothVel(case["k"], s["rho"])
        disp = s["tree"].CalcSmoothVelDisp(mean, case["k"], s["rho"])
        return mean, disp
    if kind == "points":
        nn, d2 = s["tree"].FindNearestPosPoints(s["points"], case["k"])
        rho = s["tree"].CalcDensityPosition(s["points"], case["k"])
        return {"nn": nn, "d2": d2, "rho": rho}
    raise ValueError(kind)


# ---- what a pass cannot do without

def work(case):
    """Inputs read once and outputs written once; the arithmetic of the pairs that the
    results are made of (8 operations a distance, 12 a kernel term), and for the linking
    cases of one distance per particle."""
    kind = case["kind"]
    if kind == "batch":
        lo, hi = 1.0 / case["nmin"], 1.0 / case["nmax"]
        n = case["groups"] * math.log(case["nmax"] / case["nmin"]) / (lo - hi)
        return {"bytes": 40.0 * n, "flops": 20.0 * case["k"] * n}
    n, k = case["n"], case.get("k", 0)
    if kind == "fof":
        return {"bytes": 36.0 * n, "flops": 8.0 * n}
    if kind == "knn":
        return {"bytes": (44.0 + 12.0 * k) * n, "flops": 28.0 * k * n}
    if kind == "density":
        return {"bytes": 40.0 * n, "flops": 20.0 * k * n}
    if kind == "veldensity":
        return {"bytes": 72.0 * n, "flops": 40.0 * k * n}
    if kind == "adjoint":
        return {"bytes": 80.0 * n, "flops": 60.0 * k * n}
    if kind == "fof6d":
        return {"bytes": 60.0 * n, "flops": 16.0 * n}
    if kind == "phase":
        return {"bytes": 64.0 * n, "flops": (16.0 * 8 + 32.0 * k) * n}
    if kind == "ball":
        return {"bytes": (36.0 + 4.0 * case["per_ball"]) * n, "flops": 8.0 * case["per_ball"] * n}
    if kind == "smooth":
        return {"bytes": 160.0 * n, "flops": 76.0 * k * n}
    return {"bytes": 32.0 * n + (32.0 + 12.0 * k) * case["points"],
            "flops": 28.0 * k * case["points"]}


# ---- the same in plain 64-bit torch

def _table():
    """The cubic-spline kernel table over q in [0, 2] (three dimensions)."""
    q = torch.arange(KERNRES, device=DEV, dtype=torch.float64) * (2.0 / (KERNRES - 1))
    w = torch.where(q <= 1.0, 1.0 - 0.75 * (2.0 - q) * q * q, 0.25 * (2.0 - q) ** 3)
    norm = (math.pi ** -1.5) * math.gamma(2.5) / 3.0 * 3 * 4 * 5 * 6 / (6.0 * 15.0)
    return norm * w


def _w(q, table):
    """The table interpolated linearly at q; its last entry from q = 2 on."""
    delta = 2.0 / (KERNRES - 1)
    i = (q.detach() * 0.5 * (KERNRES - 1)).to(torch.int64).clamp(0, KERNRES - 1)
    j = (i + 1).clamp_max(KERNRES - 1)
    return torch.where(i < KERNRES - 1,
                       table[i] + (table[j] - table[i]) * (q - i.to(q.dtype) * delta) / delta,
                       table[KERNRES - 1].expand_as(q))


def _blocks(pos, size):
    """Rows of point indices (-1: none), each a compact cell: halved along the widest side."""
    n = pos.shape[0]
    levels = max(0, math.ceil(math.log2(max(1.0, n / size))))
    width = -(-n // (1 << levels))
    order = torch.full(((1 << levels) * width,), -1, dtype=torch.int64, device=DEV)
    order[:n] = torch.arange(n, device=DEV)
    order = order[None]
    for _ in range(levels):
        p = pos[order.clamp_min(0)]
        real = (order >= 0)[..., None]
        span = (torch.where(real, p, -math.inf).amax(1) - torch.where(real, p, math.inf).amin(1))
        dim = span.argmax(1)
        key = p.gather(2, dim[:, None, None].expand(-1, p.shape[1], 1))[..., 0]
        key = torch.where(order >= 0, key, math.inf)
        order = order.gather(1, key.argsort(1)).reshape(order.shape[0] * 2, -1)
    return order


def _nearest(pos, k, queries=None):
    """The k nearest other particles of every particle (zero distances left out), or the k
    nearest of every query point: indices and squared distances, ascending, 64 bits."""
    n = pos.shape[0]
    own = queries is None
    q = pos if own else queries
    nn = torch.empty((q.shape[0], k), dtype=torch.int64, device=DEV)
    d2 = torch.empty((q.shape[0], k), dtype=torch.float64, device=DEV)
    cells = _blocks(pos, max(64, 2 * k))
    p = pos[cells.clamp_min(0)]
    real = (cells >= 0)[..., None]
    lo, hi = torch.where(real, p, math.inf).amin(1), torch.where(real, p, -math.inf).amax(1)
    rows = _blocks(q, 256)
    for row in rows:
        row = row[row >= 0]
        if not row.numel():
            continue
        x = q[row]
        a, b = x.amin(0), x.amax(0)

        def pairs(idx):
            y = pos[idx]
            d = (x[:, None, 0] - y[None, :, 0]) ** 2
            d += (x[:, None, 1] - y[None, :, 1]) ** 2
            d += (x[:, None, 2] - y[None, :, 2]) ** 2
            if own:
                d.masked_fill_(d == 0, math.inf)
            return d

        gap = (torch.clamp_min(lo - b, 0) + torch.clamp_min(a - hi, 0)).square().sum(1)
        # a radius that holds k neighbours of each of these queries: from the nearest cells
        close = cells[gap.topk(min(8, gap.numel()), largest=False).indices].reshape(-1)
        close = close[close >= 0]
        reach = math.inf
        if close.numel() > k + 1:
            reach = float(pairs(close).topk(k, largest=False).values[:, -1].max())
        idx = cells[gap <= reach].reshape(-1)
        idx = idx[idx >= 0]
        y = pos[idx]
        idx = idx[(torch.clamp_min(y - b, 0) + torch.clamp_min(a - y, 0)).square().sum(1) <= reach]
        got = pairs(idx).topk(k, largest=False)
        d2[row], nn[row] = got.values, idx[got.indices]
    return nn, d2


def _weights(d2, table):
    """W(r / h) / h^3 with h half the farthest of each row's distances."""
    h = 0.5 * torch.sqrt(d2[:, -1:])
    w = _w(torch.sqrt(d2[:, :-1]) / h, table)
    far = table[KERNRES - 1].expand(w.shape[0], 1)
    return torch.cat([w, far], 1) / h ** 3


def _density(nn, d2, mass, table):
    w = 0.5 * _weights(d2, table)
    rho = (w * mass[nn]).sum(1)
    return rho.index_add(0, nn.reshape(-1), (w * mass[:, None]).reshape(-1))


def exact(case, seed):
    kind = case["kind"]
    x = None
    table = _table()
    if kind in ("knn", "density", "adjoint", "smooth", "veldensity"):
        if case["n"] > 1100000:
            return None
        x = _inputs(case, seed)
        pos, mass = x["pos"], x["mass"]
        nn, d2 = _nearest(pos, case["k"])
    if kind == "knn":
        # the rows of FindNearest are in tree order: they have no value in plain torch
        return {"nn": None, "d2": None, "perm": None, "rho": _density(nn, d2, mass, table)}
    if kind == "density":
        return _density(nn, d2, mass, table)
    if kind == "veldensity":
        v = x["vel"]
        dv = (v[:, None] - v[nn]).norm(dim=2).sort(1).values
        return _density(nn, d2, mass, table), _weights(dv.square(), table).sum(1)
    if kind == "adjoint":
        pos, mass = pos.clone().requires_grad_(True), mass.clone().requires_grad_(True)
        d2 = (pos[:, None] - pos[nn]).square().sum(2)
        rho = _density(nn, d2, mass, table)
        gpos, gmass = torch.autograd.grad((x["w"] * torch.log(rho)).sum(), [pos, mass])
        return rho.detach(), gpos, gmass
    if kind == "smooth":
        v = x["vel"]
        rho = _density(nn, d2, mass, table)
        w = 0.5 * _weights(d2, table)
        to_me, to_them = w * (mass / rho)[nn], w * (mass / rho)[:, None]
        flat = nn.reshape(-1)
        mean = (to_me[..., None] * v[nn]).sum(1)
        mean = mean.index_add(0, flat, (to_them[..., None] * v[:, None]).reshape(-1, 3))
        disp = torch.zeros((case["n"], 3, 3), dtype=torch.float64, device=DEV)
        for a in range(3):
            for b in range(3):
                da, db = v[nn][..., a] - mean[:, None, a], v[nn][..., b] - mean[:, None, b]
                disp[:, a, b] += (to_me * da * db).sum(1)
                da, db = v[:, None, a] - mean[nn][..., a], v[:, None, b] - mean[nn][..., b]
                disp[:, a, b].index_add_(0, flat, (to_them * da * db).reshape(-1))
        return mean, disp
    if kind == "points":
        if case["points"] > 600000:
            return None
        x = _inputs(case, seed)
        nn, d2 = _nearest(x["pos"], case["k"], x["points"])
        # only the density: the lists hold tree indices, their distances images of the box
        rho = (_weights(d2, table) * x["mass"][nn]).sum(1)
        return {"nn": None, "d2": None, "rho": rho}
    if kind == "batch":
        if work(case)["bytes"] / 40.0 > 400000 or case["groups"] > 3000:
            return None
        x = _inputs(case, seed)
        out = torch.empty_like(x["mass"])
        off = x["off"].tolist()
        for lo, hi in zip(off[:-1], off[1:]):
            nn, d2 = _nearest(x["pos"][lo:hi], min(case["k"], hi - lo - 1))
            out[lo:hi] = _density(nn, d2, x["mass"][lo:hi], table)
        return out
    return None
