"""Cases that stand for what programs do with this framework, from one target point to the
headline catalogue: building trees, k nearest neighbours, ball and box searches, forests, and
the learned bound.  Sizes come from the benchmark's workloads and the tests, with ragged ones
between them; catalogues are drawn on the GPU from the case's seed."""
import math

import numpy as np
import torch

from cosmokdtree_b200 import forest, kdtree, learned, synth

DEV = "cuda"


def listed():
    return [
        # one galaxy looked up in a catalogue that is already on the GPU: latency of a single call
        {"name": "knn_point", "kind": "knn", "points": "uniform", "n": 1 << 20, "d": 3, "leaf": 16,
         "nq": 1, "query": "uniform", "k": 16, "sorted": True, "dtype": "f64"},
        # a drop-in program of the reference: one halo's particles as numpy arrays, a tree, and every
        # particle's neighbours back as numpy arrays
        {"name": "small_host_catalogue", "kind": "build_knn", "points": "cluster", "n": 20011, "d": 3,
         "leaf": 16, "nq": 20011, "query": "self", "k": 8, "sorted": True, "dtype": "f64",
         "host": True},
        # the plain method at its ordinary size: 10^5 targets in 2^20 uniform points, k = 16
        {"name": "knn_uniform", "kind": "knn", "points": "uniform", "n": 1 << 20, "d": 3, "leaf": 16,
         "nq": 100000, "query": "uniform", "k": 16, "sorted": True, "dtype": "f64"},
        # the headline workload: every point of a clustered periodic catalogue, k = 32
        {"name": "knn_self_clustered", "kind": "knn", "points": "clustered", "n": 1 << 24, "d": 3,
         "leaf": 16, "nq": 1 << 24, "query": "self", "k": 32, "sorted": True, "dtype": "f64"},
        # wide neighbourhoods (density profiles, smoothing kernels): k = 100, ragged sizes
        {"name": "knn_wide", "kind": "knn", "points": "clustered", "n": 1000003, "d": 3, "leaf": 16,
         "nq": 30011, "query": "self", "k": 100, "sorted": True, "dtype": "f64"},
        # phase-space neighbours: 6-D float32 catalogue, leaf 32, k = 64, particles as targets
        {"name": "knn_phase_space", "kind": "knn", "points": "phase", "n": 1 << 22, "d": 6, "leaf": 32,
         "nq": 200003, "query": "self", "k": 64, "sorted": True, "dtype": "f32"},
        # the small ball workload: 10^5 targets, radius 0.01, rows sorted by distance
        {"name": "ball_uniform", "kind": "ball", "points": "uniform", "n": 1 << 20, "d": 3, "leaf": 16,
         "nq": 100000, "query": "uniform", "r": 0.01, "sorted": True, "dtype": "f64"},
        # ball counts of a clustered catalogue at half the mean spacing: rows of very uneven length
        {"name": "ball_clustered", "kind": "ball", "points": "clustered", "n": 1 << 22, "d": 3,
         "leaf": 16, "nq": 4001, "query": "self", "r": 0.0031, "sorted": False, "dtype": "f64"},
        # the small box workload: 10^3 boxes of side 0.02
        {"name": "box_uniform", "kind": "box", "points": "uniform", "n": 1 << 20, "d": 3, "leaf": 16,
         "nq": 1000, "side": 0.02, "dtype": "f64"},
        # a forest of independent halos built together and a tenth of each one's particles searched
        {"name": "forest_nfw", "kind": "forest", "trees": 200, "n_lo": 1000, "n_hi": 1000000, "leaf": 16,
         "k": 8, "box": True},
        # a snapshot arrives, its tree is built, and some targets are looked up in it
        {"name": "build_snapshot", "kind": "build_knn", "points": "clustered", "n": 1 << 24, "d": 3,
         "leaf": 16, "nq": 100003, "query": "mixed", "k": 16, "sorted": True, "dtype": "f64",
         "host": False},
        # the learned bound on targets drawn half from the particles, half uniformly
        {"name": "knn_learned", "kind": "learned", "points": "clustered", "n": 1 << 22, "d": 3,
         "leaf": 16, "nq": 1000000, "query": "mixed", "k": 32, "sorted": True, "dtype": "f64"},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["knn", "knn", "knn", "build_knn", "build_knn", "ball", "box", "forest", "learned"])
    if kind == "forest":
        return {"kind": kind, "trees": _log(rng, 3, 200), "n_lo": 1000, "n_hi": _log(rng, 3000, 1000000),
                "leaf": rng.choice([8, 16, 32]), "k": rng.choice([1, 4, 8, 16, 31]),
                "box": rng.random() < 0.7}
    points = rng.choice(["uniform", "uniform", "clustered", "clustered", "cluster", "phase"])
    if kind in ("ball", "box", "learned") and points == "phase":
        points = "clustered"
    d = 6 if points == "phase" else rng.choice([2, 3, 3, 3]) if points == "uniform" else 3
    c = {"kind": kind, "points": points, "d": d, "leaf": 32 if d == 6 else rng.choice([8, 16, 16, 32]),
         "dtype": "f32" if d == 6 else rng.choice(["f64", "f64", "f32"])}
    if kind == "knn":
        c["n"] = _log(rng, 5000, 1 << 22)
        c["k"] = rng.choice([1, 5, 8, 16, 32, 48, 64, 65, 100, 128])
        most = (1 << 25) // c["k"] // (8 if d == 6 else 1)
        c["nq"] = _log(rng, 1, min(1 << 20, most))
        c["query"] = rng.choice(["self", "uniform", "mixed"]) if points != "phase" else "self"
        c["sorted"] = rng.random() < 0.8
    elif kind == "build_knn":
        c["n"] = _log(rng, 2000, 1 << 23)
        c["k"] = rng.choice([1, 8, 16, 32])
        c["nq"] = _log(rng, 100, 100000)
        c["query"] = "self"
        c["sorted"] = True
        c["host"] = c["n"] < 100000 and rng.random() < 0.5
    elif kind == "ball":
        c["n"] = _log(rng, 20000, 1 << 22)
        if points == "uniform":  # a mean count of 1 to 100 a row
            c["nq"] = _log(rng, 1, 100000)
            hits = math.exp(rng.uniform(0.0, math.log(100.0)))
            ball = math.pi if d == 2 else 4.0 * math.pi / 3.0
            c["r"] = (hits / (c["n"] * ball)) ** (1.0 / d)
        else:
            c["nq"] = _log(rng, 1, 4001)
            c["r"] = rng.uniform(0.2, 0.5) * c["n"] ** (-1.0 / 3.0)
        c["query"] = rng.choice(["self", "uniform"])
        c["sorted"] = rng.random() < 0.5 if points == "uniform" else rng.random() < 0.2
    elif kind == "box":
        c["n"] = _log(rng, 20000, 1 << 22)
        c["nq"] = _log(rng, 1, 20000)
        c["side"] = (math.exp(rng.uniform(0.0, math.log(200.0))) / c["n"]) ** (1.0 / d)
    else:
        c["n"] = _log(rng, 100000, 1 << 22)
        c["nq"] = _log(rng, 20000, 1000000)
        c["k"] = rng.choice([8, 16, 32, 64])
        c["query"] = "mixed"
        c["sorted"] = True
    return c


# ------------------------------------------------------------------ catalogues

def _rng(seed, part):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1000003 + part)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _wrap(p):
    p = torch.remainder(p + 0.5, 1.0) - 0.5
    return torch.where(p >= 0.5, torch.full_like(p, -0.5), p)


def _nfw(g, conc, rvir):
    """Positions about the centre of NFW-like clusters, one per point."""
    mu = lambda y: torch.log1p(y) - y / (1.0 + y)  # noqa: E731
    n = conc.shape[0]
    target = _rand(g, n) * mu(conc)
    lo, hi = torch.zeros_like(conc), torch.ones_like(conc)
    for _ in range(36):
        mid = 0.5 * (lo + hi)
        below = mu(conc * mid) < target
        lo = torch.where(below, mid, lo)
        hi = torch.where(below, hi, mid)
    v = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    return (0.5 * (lo + hi) * rvir / torch.linalg.norm(v, dim=1))[:, None] * v


def _clustered(g, n, labels=False):
    """70 % of the points in 4096 NFW-like clusters of a periodic unit box, 30 % background."""
    m = 4096
    centre = _rand(g, m, 3) - 0.5
    conc = 5.0 + 10.0 * _rand(g, m)
    rvir = 0.002 * 10.0 ** _rand(g, m)
    a = -0.9
    mass = (1.0 + _rand(g, m) * (1e4 ** a - 1.0)) ** (1.0 / a)
    nc = int(round(0.7 * n))
    lab = torch.searchsorted(torch.cumsum(mass, 0) / mass.sum(), _rand(g, nc)).clamp_max(m - 1)
    pos = _wrap(centre[lab] + _nfw(g, conc[lab], rvir[lab]))
    p = torch.cat([pos, _rand(g, n - nc, 3) - 0.5])
    perm = torch.randperm(n, generator=g, device=DEV)
    if not labels:
        return p[perm].contiguous()
    lab = torch.cat([lab, torch.full((n - nc,), -1, device=DEV, dtype=lab.dtype)])
    return p[perm], lab[perm]


def _points(case, seed):
    g, n, d = _rng(seed, 1), case["n"], case["d"]
    if case["points"] == "uniform":
        p = _rand(g, n, d)
    elif case["points"] == "cluster":
        p = _wrap(_nfw(g, torch.full((n,), 4.0, device=DEV, dtype=torch.float64) + 16.0 * _rand(g, 1), 0.25))
    elif case["points"] == "clustered":
        p = _clustered(g, n)
    else:  # positions and velocities: each cluster has a bulk velocity and a dispersion
        x, lab = _clustered(g, n, labels=True)
        sigma = 0.05 + 0.25 * _rand(g, 4096)
        bulk = 0.1 * torch.randn(4096, 3, generator=g, device=DEV, dtype=torch.float64)
        v = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
        v = torch.where((lab >= 0)[:, None], bulk[lab] + v * sigma[lab][:, None], 0.1 * v)
        p = torch.cat([x, v], 1)
    return p.to(torch.float32 if case["dtype"] == "f32" else torch.float64).contiguous()


def _box(case):
    return 1.0 if case["points"] in ("clustered", "cluster") else None


def _targets(case, p, seed):
    g, nq, q = _rng(seed, 2), case["nq"], case["query"]
    if q == "self" and nq == case["n"]:
        return p.to(torch.float64)
    own = p[torch.randint(0, case["n"], (nq,), generator=g, device=DEV)].to(torch.float64)
    if q == "self":
        return own
    flat = _rand(g, nq, case["d"])
    if case["points"] == "phase":
        flat = flat - 0.5
    elif _box(case):
        flat = flat - 0.5
    if q == "uniform":
        return flat
    return torch.where(_rand(g, nq, 1) < 0.5, own, flat).contiguous()


def _boxes(case, p, seed):
    g = _rng(seed, 3)
    c = _rand(g, case["nq"], case["d"]) - (0.5 if _box(case) else 0.0)
    h = 0.5 * case["side"]
    return torch.stack([c - h, c + h], dim=2).reshape(case["nq"], -1).contiguous()


# The rows of ball, box and forest results have the lengths that the geometry gives them.  Their
# catalogue is therefore the same for every seed up to the order of its points, the order of its
# targets and the order of its axes, which the seed draws.
GEOMETRY = 11


def _axes(seed, d):
    return torch.randperm(d, generator=_rng(seed, 5), device=DEV)


def _shuffled(case, seed):
    p = _points(case, GEOMETRY)
    x = _boxes(case, p, GEOMETRY) if case["kind"] == "box" else _targets(case, p, GEOMETRY)
    g, ax = _rng(seed, 6), _axes(seed, case["d"])
    p = p[torch.randperm(case["n"], generator=g, device=DEV)][:, ax].contiguous()
    x = x[torch.randperm(case["nq"], generator=g, device=DEV)]
    x = x.reshape(case["nq"], case["d"], -1)[:, ax].reshape(case["nq"], -1).contiguous()
    return p, x


def _forest(case, seed):
    p, off = synth.forest_catalogue(case["trees"], seed=GEOMETRY, n_range=(case["n_lo"], case["n_hi"]))
    g = _rng(GEOMETRY, 4)
    nq = np.maximum(1, np.diff(off) // 10)
    qoff = np.concatenate([[0], np.cumsum(nq)]).astype(np.int64)
    tree = torch.repeat_interleave(torch.arange(case["trees"], device=DEV),
                                   torch.from_numpy(nq).to(DEV))
    o = torch.from_numpy(off).to(DEV)
    pick = o[tree] + (_rand(g, int(qoff[-1])) * (o[tree + 1] - o[tree])).long()
    q = p[pick].contiguous()
    boxes = boff = None
    if case["box"]:
        nb = 64
        c = p[(o[:-1, None] + (_rand(g, case["trees"], nb) * (o[1:] - o[:-1])[:, None]).long()).reshape(-1)]
        boxes = torch.stack([c - 0.025, c + 0.025], dim=2).reshape(-1, 6).contiguous()
        boff = np.arange(0, nb * case["trees"] + 1, nb, dtype=np.int64)
        boxes = boxes.reshape(-1, 3, 2)[:, _axes(seed, 3)].reshape(-1, 6).contiguous()
    tree = torch.repeat_interleave(torch.arange(case["trees"], device=DEV), o[1:] - o[:-1])
    by = torch.argsort(tree + _rand(_rng(seed, 6), p.shape[0]))  # another order within each tree
    p, q = p[by][:, _axes(seed, 3)].contiguous(), q[:, _axes(seed, 3)].contiguous()
    return p, off, q, qoff, boxes, boff


def prepare(case, seed):
    if case["kind"] == "forest":
        p, off, q, qoff, boxes, boff = _forest(case, seed)
        return {"case": case, "p": p, "off": off, "q": q, "qoff": qoff, "boxes": boxes, "boff": boff}
    s = {"case": case}
    if case["kind"] in ("ball", "box"):
        p, x = _shuffled(case, seed)
        s["tree"] = kdtree.build_kdtree(p, leaf=case["leaf"], boxsize=_box(case))
        s["boxes" if case["kind"] == "box" else "q"] = x
        return s
    p = _points(case, seed)
    if case["kind"] == "build_knn":
        q = _targets(case, p, seed)
        s["p"], s["q"] = (p.cpu().numpy(), q.cpu().numpy()) if case["host"] else (p, q)
        return s
    s["tree"] = kdtree.build_kdtree(p, leaf=case["leaf"], boxsize=_box(case))
    s["q"] = _targets(case, p, seed)
    if case["kind"] == "learned":  # a network trained once, kept beside the tree
        s["net"] = learned.LearnedBound(seed=seed)
        train = dict(case, nq=30000)
        s["net"].fit(s["tree"], _targets(train, p, seed + 7919), case["k"], epochs=8, batch=1024)
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    c = s["case"]
    if c["kind"] == "knn":
        return kdtree.knn_search(s["tree"], s["q"], c["k"], sorted=c["sorted"])
    if c["kind"] == "build_knn":
        tree = kdtree.build_kdtree(s["p"], leaf=c["leaf"], boxsize=_box(c))
        out = kdtree.knn_search(tree, s["q"], c["k"], sorted=c["sorted"])
        kdtree.deallocate_kdtree(tree)
        return out
    if c["kind"] == "ball":
        return kdtree.ball_search_csr(s["tree"], s["q"], c["r"], sorted=c["sorted"])
    if c["kind"] == "box":
        return kdtree.box_search_csr(s["tree"], s["boxes"])
    if c["kind"] == "learned":
        return s["net"].knn(s["tree"], s["q"], c["k"], sorted=c["sorted"])
    f = forest.build_forest(s["p"], s["off"], leaf=c["leaf"], boxsize=1.0)
    out = f.knn(s["q"], s["qoff"], c["k"])
    if c["box"]:
        out = out + f.box_csr(s["boxes"], s["boff"])
    f.close()
    return out


def _mean_points(c):
    a, b = math.log(c["n_lo"]), math.log(c["n_hi"])
    return (c["n_hi"] - c["n_lo"]) / (b - a)


def work(case):
    """Each input coordinate read once, each result written once.  A search that does not ask for all of a
    tree's points reads at least those that it returns."""
    c = case
    if c["kind"] == "forest":
        n = c["trees"] * _mean_points(c)
        nq = 0.1 * n
        by = n * 24 + n * 28 + nq * 24 + nq * c["k"] * 16
        return {"bytes": by, "flops": nq * c["k"] * 9 + 6 * n}
    d, n, nq = c["d"], c["n"], c["nq"]
    item = 4 if c["dtype"] == "f32" else 8
    if c["kind"] in ("knn", "learned"):
        return {"bytes": min(n, nq * c["k"]) * d * 8 + nq * d * 8 + nq * c["k"] * 16,
                "flops": nq * c["k"] * 3 * d}
    if c["kind"] == "build_knn":
        by = n * d * item + n * (8 * d + 4) + nq * d * 8 + nq * c["k"] * 16
        return {"bytes": by, "flops": 2 * d * n + nq * c["k"] * 3 * d}
    vol = (2 * c["r"]) ** d if c["kind"] == "ball" else c["side"] ** d
    hits = nq * min(n, max(1.0, n * vol))
    if c["kind"] == "ball":
        if c["points"] != "uniform":  # most targets sit in clusters some thousands of times the mean density
            hits = nq * min(n, 50000.0)
        return {"bytes": min(n, hits) * d * 8 + nq * d * 8 + hits * 16, "flops": hits * 3 * d}
    return {"bytes": min(n, hits) * d * 8 + nq * 2 * d * 8 + hits * 8, "flops": hits * 2 * d}


# ------------------------------------------------------------------ in 64 bits

def _d2(p, q, box):
    s = None
    for j in range(p.shape[1]):
        dx = (p[None, :, j] - q[:, None, j]).abs()
        if box:
            dx = torch.minimum(dx, box - dx)
        s = dx * dx if s is None else s + dx * dx
    return s


def exact(case, seed):
    """Brute force in 64 bits: distances only (ids are whole numbers)."""
    c = case
    if c["kind"] in ("box", "forest") or (c["kind"] != "ball" and not c["sorted"]):
        return None
    if c["kind"] == "ball" and (not c["sorted"] or c["points"] != "uniform"):
        return None
    if c["n"] * c["nq"] * c["d"] > 4e11:
        return None
    if c["kind"] == "ball":
        p, q = _shuffled(c, seed)
    else:
        p = _points(c, seed)
        q = _targets(c, p, seed)
    p = p.to(torch.float64)
    rows = max(1, (1 << 27) // c["n"])
    got = []
    for a in range(0, c["nq"], rows):
        s = _d2(p, q[a:a + rows], _box(c))
        if c["kind"] == "ball":
            hit = (s <= c["r"] * c["r"]).nonzero()
            v = s[hit[:, 0], hit[:, 1]]
            by = torch.argsort(v, stable=True)
            by = by[torch.argsort(hit[by, 0], stable=True)]
            got.append(torch.sqrt(v[by]))
        else:
            k = min(c["k"], c["n"])
            v = torch.sqrt(torch.topk(s, k, dim=1, largest=False, sorted=True).values)
            got.append(v)
    dist = torch.cat(got)
    if c["kind"] == "ball":
        return (None, None, dist)
    return (dist.cpu().numpy() if c.get("host") else dist, None)
