"""The workloads by which this package's speed is followed, over its public entry points.

A case is a dict of plain values. `listed()` gives the fixed ones, `draw(rng)`
one more of the same ranges, `prepare(case, seed)` the inputs a caller holds
before the call, `run(state)` one pass, `work(case)` the bytes and operations a
pass cannot do without and `exact(case, seed)` the same outputs in float64 by
plain torch.

Clouds: "scene" is the outdoor composition of the benchmark (ground plane with
1 cm noise, vertical walls, cylinders, uniform scatter, shuffled) in a box of
`side` x `side` x side / 5 metres; "uniform" fills a cube of edge `side`, as the
reference's own benchmarks do.
"""

import math

import numpy as np
import torch

import point_geometric_features_gb300 as pgeof

DEVICE = "cuda"
REQUEST = "Verticality,Curvature,Planarity,Normal_z"  # the serving stream's feature list


# ------------------------------------------------------------------ cases
def listed():
    return [
        # The smallest calls: a 10k-point uniform cube with k = 20, where launches and latency count. One call
        # for the neighbours, one for the features.
        {"name": "knn small", "kind": "knn", "cloud": "uniform", "n": 10_000, "m": 0, "k": 20, "side": 1.0},
        {"name": "features small", "kind": "features", "cloud": "uniform", "n": 10_000, "k": 20, "scales": "",
         "side": 1.0},
        # The reference's benchmark of selected features: float64 points, sparse neighbourhoods.
        {"name": "selected f64", "kind": "selected", "cloud": "uniform", "n": 10_000, "side": 200.0, "radius": 5.0,
         "k": 50, "ids": "Verticality", "dtype": "float64", "host": False},
        # One request of the serving stream: a mid-size cloud in host memory, results back in host memory.
        {"name": "selected request", "kind": "selected", "cloud": "scene", "n": 20_011, "side": 20.0, "radius": 0.0,
         "k": 32, "ids": REQUEST, "dtype": "float32", "host": True},
        # Queries that are not the data: labels or features carried from one cloud to another.
        {"name": "knn queries", "kind": "knn", "cloud": "scene", "n": 400_009, "m": 100_003, "k": 16, "side": 70.0},
        # The benchmark's scene: k = 50 neighbours of a million points, and the three-scale features over them.
        {"name": "knn scene", "kind": "knn", "cloud": "scene", "n": 1_000_000, "m": 0, "k": 50, "side": 100.0},
        {"name": "multiscale scene", "kind": "features", "cloud": "scene", "n": 1_000_000, "k": 50,
         "scales": "10,20,50", "side": 100.0},
        # Float64 clouds (surveyed coordinates) through the float64 feature pass.
        {"name": "features f64", "kind": "features_f64", "cloud": "scene", "n": 200_003, "k": 32, "scales": "",
         "side": 45.0},
        # Radius neighbourhoods of a large scan, and the optimal size of each over the CSR of such neighbourhoods.
        {"name": "radius scene", "kind": "radius", "cloud": "scene", "n": 4_000_000, "side": 100.0, "radius": 0.5,
         "k": 64},
        {"name": "optimal", "kind": "optimal", "cloud": "scene", "n": 4_000_000, "side": 100.0, "radius": 0.5, "k": 64,
         "k_min": 1, "k_step": 1, "k_min_search": 10},
        # Features only, neighbours and features in one call, of a cloud of odd size.
        {"name": "knn features", "kind": "knn_features", "cloud": "scene", "n": 3_000_017, "k": 32, "scales": "16,32",
         "side": 170.0},
        # Many clouds of uneven size (log-uniform 2k to 200k points) through one plan.
        {"name": "batch", "kind": "batch", "clouds": 256, "lo": 2_000, "hi": 200_000, "k": 32, "sizes_seed": 3},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scene_side(rng, n):
    """A side that gives the scene between 25 and 400 points per square metre of its plan."""
    return round(math.sqrt(n / math.exp(rng.uniform(math.log(25.0), math.log(400.0)))), 2)


def draw(rng):
    kind = rng.choice(["knn", "knn", "knn queries", "features", "features", "features_f64", "selected",
                       "selected request", "radius", "optimal", "knn_features", "batch"])
    cloud = rng.choice(["scene", "scene", "uniform"])
    k = rng.choice([8, 10, 16, 20, 25, 32, 50, 64, 100])

    def side(n):
        return _scene_side(rng, n) if cloud == "scene" else 1.0

    if kind in ("knn", "knn queries"):
        n = _log_uniform(rng, 1_000, 3_000_000)
        m = _log_uniform(rng, 1_000, 1_000_000) if kind == "knn queries" else 0
        return {"kind": "knn", "cloud": cloud, "n": n, "m": m, "k": k, "side": side(n)}
    if kind == "features":
        n = _log_uniform(rng, 1_000, 10_000_000)
        k = min(k, 50 if n < 3_000_000 else 20)
        scales = rng.choice(["", "", "%d" % max(1, k // 2), "%d,%d" % (max(1, k // 2), k),
                             "%d,%d,%d" % (max(1, k // 4), max(1, k // 2), k)])
        return {"kind": "features", "cloud": cloud, "n": n, "k": k, "scales": scales, "side": side(n)}
    if kind == "features_f64":
        n = _log_uniform(rng, 1_000, 1_000_000)
        k = min(k, 50)
        scales = rng.choice(["", "", "%d,%d" % (max(3, k // 2), k)])
        return {"kind": "features_f64", "cloud": cloud, "n": n, "k": k, "scales": scales, "side": side(n)}
    if kind == "selected":
        n = _log_uniform(rng, 1_000, 500_000)
        return {"kind": "selected", "cloud": cloud, "n": n, "side": side(n), "radius": 0.0, "k": rng.choice([16, 32, 50, 64]),
                "ids": rng.choice(["Verticality", REQUEST]), "dtype": rng.choice(["float32", "float64"]), "host": False}
    if kind == "selected request":
        n = _log_uniform(rng, 1_000, 500_000)
        cloud = "scene"
        return {"kind": "selected", "cloud": cloud, "n": n, "side": side(n), "radius": 0.0, "k": rng.choice([16, 32, 64]),
                "ids": REQUEST, "dtype": "float32", "host": True}
    if kind == "radius":
        n = _log_uniform(rng, 10_000, 3_000_000)
        cloud = "scene"
        s = side(n)
        return {"kind": "radius", "cloud": cloud, "n": n, "side": s,
                "radius": round(_disc_radius(n, s, rng.uniform(0.5, 2.0) * 40), 4), "k": rng.choice([30, 50, 64])}
    if kind == "optimal":
        n = _log_uniform(rng, 10_000, 3_000_000)
        cloud = "scene"
        s = side(n)
        return {"kind": "optimal", "cloud": cloud, "n": n, "side": s,
                "radius": round(_disc_radius(n, s, rng.uniform(0.5, 2.0) * 40), 4), "k": rng.choice([30, 50, 64]),
                "k_min": 1, "k_step": rng.choice([1, 1, 2, 5]), "k_min_search": 10}
    if kind == "knn_features":
        n = _log_uniform(rng, 1_000, 3_000_000)
        k = min(k, 64)
        scales = rng.choice(["", "%d,%d" % (max(1, k // 2), k), "%d,%d,%d" % (max(1, k // 4), max(1, k // 2), k)])
        return {"kind": "knn_features", "cloud": cloud, "n": n, "k": k, "scales": scales, "side": side(n)}
    return {"kind": "batch", "clouds": _log_uniform(rng, 2, 200), "lo": 2_000, "hi": 200_000, "k": rng.choice([16, 20, 32]),
            "sizes_seed": rng.randrange(1_000_000)}


# ------------------------------------------------------------------ inputs
def _disc_radius(n, side, count):
    """The radius of a disc that holds `count` points of the scene's ground (half its points on side x side)."""
    return math.sqrt(count * side * side / (math.pi * 0.5 * n))


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _uniform(n, side, g, dtype=torch.float32):
    return torch.rand((n, 3), generator=g, device=DEVICE, dtype=dtype) * side


def _scene(n, side, g, dtype=torch.float32):
    """50% ground, 25% on vertical walls, 15% on vertical cylinders, 10% scatter, shuffled."""
    height = 0.2 * side
    walls = max(2, int(round(40 * (side / 100.0) ** 2)))
    poles = max(2, int(round(200 * (side / 100.0) ** 2)))

    def u(size, lo=0.0, hi=1.0):
        return torch.rand(size, generator=g, device=DEVICE, dtype=torch.float64) * (hi - lo) + lo

    def normal(size, sigma):
        return torch.randn(size, generator=g, device=DEVICE, dtype=torch.float64) * sigma

    n_wall, n_pole, n_scatter = int(0.25 * n), int(0.15 * n), int(0.10 * n)
    n_ground = n - n_wall - n_pole - n_scatter
    ground = torch.stack([u(n_ground, 0, side), u(n_ground, 0, side), normal(n_ground, 0.01)], 1)
    length, tall, angle = u(walls, 0.05, 0.3) * side, u(walls, 0.15, 0.75) * height, u(walls, 0, math.pi)
    cx, cy = u(walls) * (side - length) + 0.5 * length, u(walls) * (side - length) + 0.5 * length
    w = torch.multinomial(length * tall, n_wall, replacement=True, generator=g)
    along, off = u(n_wall, -0.5, 0.5) * length[w], normal(n_wall, 0.005)
    wall = torch.stack([cx[w] + along * torch.cos(angle[w]) - off * torch.sin(angle[w]),
                        cy[w] + along * torch.sin(angle[w]) + off * torch.cos(angle[w]), u(n_wall) * tall[w]], 1)
    radius, tall = u(poles, 0.1, 0.5), u(poles, 2.0, 10.0) * (height / 20.0)
    cx, cy = u(poles) * (side - 2 * radius) + radius, u(poles) * (side - 2 * radius) + radius
    p = torch.multinomial(radius * tall, n_pole, replacement=True, generator=g)
    theta = u(n_pole, 0, 2 * math.pi)
    pole = torch.stack([cx[p] + radius[p] * torch.cos(theta), cy[p] + radius[p] * torch.sin(theta), u(n_pole) * tall[p]], 1)
    scatter = u((n_scatter, 3)) * torch.tensor([side, side, height], device=DEVICE, dtype=torch.float64)
    xyz = torch.cat([ground, wall, pole, scatter])
    return xyz[torch.randperm(n, generator=g, device=DEVICE)].to(dtype).contiguous()


def _cloud(case, seed, n=None, dtype=torch.float32):
    g = _generator(seed)
    make = _scene if case["cloud"] == "scene" else _uniform
    return make(case["n"] if n is None else n, case["side"], g, dtype)


def _batch_clouds(case, seed):
    rng = np.random.default_rng(case["sizes_seed"])
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["clouds"])).astype(np.int64)
    sides = rng.uniform(5.0, 50.0, case["clouds"])
    g = _generator(seed)
    return [_scene(int(n), float(s), g) for n, s in zip(sizes, sides)]


def _scales(case):
    return [int(v) for v in case["scales"].split(",")] if case["scales"] else None


def _radius(case):
    return case["radius"] or (_disc_radius(case["n"], case["side"], 1.5 * case["k"]) if case["cloud"] == "scene" else
                              case["side"] * (1.5 * case["k"] / (case["n"] * 4.19)) ** (1 / 3))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "plan": pgeof.BatchPlan(_batch_clouds(case, seed), case["k"])}
    if kind == "selected":
        xyz = _cloud(case, seed, dtype=getattr(torch, case["dtype"]))
        return {"kind": kind, "xyz": xyz.cpu().numpy() if case["host"] else xyz, "radius": _radius(case), "k": case["k"],
                "ids": [getattr(pgeof.EFeatureID, v) for v in case["ids"].split(",")]}
    xyz = _cloud(case, seed)
    state = {"kind": kind, "xyz": xyz, "k": case["k"]}
    if kind == "knn":
        state["query"] = _cloud(case, seed + 77_000, case["m"]) if case["m"] else xyz
    elif kind in ("features", "features_f64"):
        # the neighbour lists a caller of the feature passes comes with
        idx, _ = pgeof.knn_search(xyz, xyz, case["k"])
        state["nn"] = idx.view(torch.int32).reshape(-1)
        state["ptr"] = torch.arange(0, case["k"] * (case["n"] + 1), case["k"], dtype=torch.int32, device=DEVICE)
        state["scales"] = _scales(case)
        if kind == "features_f64":
            state["xyz"] = xyz.double() + 1.0e3  # surveyed coordinates keep an offset that float32 would round
    elif kind == "radius":
        state["radius"] = case["radius"]
    elif kind == "optimal":
        state["nn"], state["ptr"] = pgeof.radius_search_csr(xyz, xyz, case["radius"], case["k"])
        state["args"] = (case["k_min"], case["k_step"], case["k_min_search"])
    elif kind == "knn_features":
        state["scales"] = _scales(case)
    return state


# ------------------------------------------------------------------ a pass
def run(state):
    kind = state["kind"]
    if kind == "knn":
        idx, d2 = pgeof.knn_search(state["xyz"], state["query"], state["k"])
        return idx.view(torch.int32), d2
    if kind == "features":
        if state["scales"]:
            return pgeof.compute_features_multiscale(state["xyz"], state["nn"], state["ptr"], state["scales"], check=False)
        return pgeof.compute_features(state["xyz"], state["nn"], state["ptr"], check=False)
    if kind == "features_f64":
        if state["scales"]:
            return pgeof.compute_features_multiscale_f64(state["xyz"], state["nn"], state["ptr"], state["scales"], check=False)
        return pgeof.compute_features_f64(state["xyz"], state["nn"], state["ptr"], check=False)
    if kind == "selected":
        return pgeof.compute_features_selected(state["xyz"], state["radius"], state["k"], state["ids"])
    if kind == "radius":
        return pgeof.radius_search(state["xyz"], state["xyz"], state["radius"], state["k"])
    if kind == "optimal":
        return pgeof.compute_features_optimal(state["xyz"], state["nn"], state["ptr"], *state["args"], check=False)
    if kind == "knn_features":
        return pgeof.knn_features(state["xyz"], state["k"], state["scales"])
    idx, d2, features = state["plan"]()
    return idx.view(torch.int32), d2, features


def work(case):
    """Inputs read once and outputs written once; operations: 8 per neighbour's distance, 18 per neighbour of a
    covariance, 1000 per eigen-decomposition with its features, 60 per candidate size of the optimal scan."""
    kind, k = case["kind"], case["k"]
    if kind == "batch":
        rng = np.random.default_rng(case["sizes_seed"])
        n = int(np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["clouds"])).astype(np.int64).sum())
        return {"bytes": n * (12 + 8 * k + 44), "flops": n * (8 * k + 18 * k + 1000)}
    n = case["n"]
    if kind == "knn":
        m = case["m"] or n
        return {"bytes": 12 * n + (12 * m if case["m"] else 0) + 8 * m * k, "flops": 8 * m * k}
    if kind in ("features", "features_f64"):
        s = len(_scales(case) or [0])
        size = 4 if kind == "features" else 8
        return {"bytes": n * (3 * size + 4 * k + 4 + 11 * s * size), "flops": n * (18 * k + 1000 * s)}
    if kind == "knn_features":
        s = len(_scales(case) or [0])
        return {"bytes": n * (12 + 44 * s), "flops": n * (26 * k + 1000 * s)}
    if kind == "selected":
        size = 4 if case["dtype"] == "float32" else 8
        ids = len(case["ids"].split(","))
        rows = min(k, _mean_hits(case))
        return {"bytes": n * size * (3 + ids), "flops": n * (26 * rows + 1000)}
    rows = min(k, _mean_hits(case))
    if kind == "radius":
        return {"bytes": n * (12 + 8 * k), "flops": n * 8 * rows}
    return {"bytes": n * (12 + 4 * rows + 4 + 48), "flops": n * (18 * rows + 60 * rows / case["k_step"] + 1000)}


def _mean_hits(case):
    """Points inside the search radius around an average point, roughly."""
    n, r, side = case["n"], _radius(case), case["side"]
    return 0.5 * n * math.pi * (r / side) ** 2 if case["cloud"] == "scene" else n * 4.19 * (r / side) ** 3


# ------------------------------------------------------------------ the same in float64
PAIRS = 6e10  # distances that a brute-force search may take


def _search64(data, query, k, radius=None):
    """The k nearest of each query by distances in the data's own type (nearest first); `radius` drops those at or
    beyond it. Returns (indices, hits)."""
    idx = torch.empty((query.shape[0], k), dtype=torch.int64, device=data.device)
    hits = torch.full((query.shape[0],), k, dtype=torch.int64, device=data.device)
    step = max(1, int(4e8 / data.shape[0]))
    for a in range(0, query.shape[0], step):
        q = query[a:a + step]
        d = torch.zeros((q.shape[0], data.shape[0]), dtype=data.dtype, device=data.device)
        for c in range(3):
            t = q[:, c, None] - data[None, :, c]
            d += t * t
        near, at = torch.topk(d, k, dim=1, largest=False, sorted=True)
        idx[a:a + step] = at
        if radius is not None:
            r2 = torch.tensor(radius, dtype=data.dtype, device=data.device) ** 2
            hits[a:a + step] = (near < r2).sum(1)
    return idx, hits


def _eigh3(cov):
    """Eigenvalues (ascending) and eigenvectors (columns) of symmetric (n, 3, 3) matrices by cyclic Jacobi."""
    a = cov.clone()
    v = torch.eye(3, dtype=a.dtype, device=a.device).expand_as(a).clone()
    for _ in range(9):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            apq = a[:, p, q]
            theta = (a[:, q, q] - a[:, p, p]) / torch.where(apq == 0, torch.ones_like(apq), 2 * apq)
            sign = torch.where(theta < 0, -torch.ones_like(theta), torch.ones_like(theta))
            t = torch.where(apq == 0, torch.zeros_like(apq), sign / (theta.abs() + torch.sqrt(theta * theta + 1)))
            c = 1 / torch.sqrt(t * t + 1)
            s = t * c
            for m in (a, v):  # columns of both, then rows of a
                x, y = m[:, :, p].clone(), m[:, :, q].clone()
                m[:, :, p], m[:, :, q] = c[:, None] * x - s[:, None] * y, s[:, None] * x + c[:, None] * y
            x, y = a[:, p, :].clone(), a[:, q, :].clone()
            a[:, p, :], a[:, q, :] = c[:, None] * x - s[:, None] * y, s[:, None] * x + c[:, None] * y
    w, order = torch.sort(torch.diagonal(a, dim1=1, dim2=2), dim=1, stable=True)
    return w, torch.gather(v, 2, order[:, None, :].expand_as(v))


def _pca64(points, mask):
    """Clamped eigenvalues and eigenvectors of the masked neighbourhoods, (rows, k, 3) with (rows, k)."""
    m = mask.to(torch.float64)[:, :, None]
    count = m.sum(1).clamp(min=1)
    centred = (points - (points * m).sum(1, keepdim=True) / count[:, None, :]) * m
    w, v = _eigh3(torch.einsum("rki,rkj->rij", centred, centred) / count[:, :, None])
    flip = torch.where(v[:, 2:3, 2:3] < 0, -1.0, 1.0).to(v.dtype)
    return w.clamp(min=0), torch.cat([v[:, :, :2], v[:, :, 2:] * flip], 2)


def _features64(w, v):
    """The eleven features of each neighbourhood, in their order, from ascending eigenvalues and their vectors."""
    s0, s1, s2 = torch.sqrt(w).unbind(1)
    f = 1 / (s0 + 1e-3)
    u = (w[:, None, :] * v.abs()).sum(2)
    norm = torch.linalg.norm(u, dim=1)
    verticality = torch.where(s0 > 0, u[:, 2] / torch.where(norm > 0, norm, torch.ones_like(norm)), torch.zeros_like(s0))
    return torch.stack([(s0 - s1) * f, (s1 - s2) * f, s2 * f, verticality, v[:, 0, 2], v[:, 1, 2], v[:, 2, 2], s0,
                        torch.sqrt(s0 * s1 + 1e-6), (s0 * s1 * s2 + 1e-9) ** (1 / 3), s2 / (s0 + s1 + s2 + 1e-3)], 1)


def _rows64(xyz, nn, sizes, chunk=1 << 17):
    """Features (rows, 11) of the first sizes[i] entries of nn[i]; rows of size 0 are 0."""
    out = torch.zeros((nn.shape[0], 11), dtype=torch.float64, device=xyz.device)
    place = torch.arange(nn.shape[1], device=xyz.device)
    for a in range(0, nn.shape[0], chunk):
        n = sizes[a:a + chunk]
        f = _features64(*_pca64(xyz[nn[a:a + chunk]].double(), place[None, :] < n[:, None]))
        out[a:a + chunk] = torch.where(n[:, None] > 0, f, torch.zeros_like(f))
    return out


def _full(rows, size):
    return torch.full((rows,), size, dtype=torch.int64, device=DEVICE)


def _exact_optimal(case, seed):
    s = prepare(case, seed)
    xyz, ptr = s["xyz"].double(), s["ptr"].view(torch.int32).long()
    size = ptr[1:] - ptr[:-1]
    n, width = size.shape[0], case["k"]
    flat = s["nn"].view(torch.int32).long()
    k0 = max(case["k_min"], case["k_min_search"])
    best = torch.full((n,), math.inf, dtype=torch.float64, device=DEVICE)
    k_opt = torch.zeros(n, dtype=torch.int64, device=DEVICE)
    first = xyz[flat[ptr[:-1].clamp(max=max(flat.shape[0] - 1, 0))]]
    s1 = torch.zeros((n, 3), dtype=torch.float64, device=DEVICE)
    s2 = torch.zeros((n, 3, 3), dtype=torch.float64, device=DEVICE)
    for k in range(1, width + 1):
        live = size >= k
        d = torch.where(live[:, None], xyz[flat[(ptr[:-1] + k - 1).clamp(max=flat.shape[0] - 1)]] - first, 0.0)
        s1 += d
        s2 += d[:, :, None] * d[:, None, :]
        use = live & (size >= k0) & (k >= k0) & ((size == k) | (k == k0) | (k % case["k_step"] == 0))
        mean = s1 / k
        w = _eigenvalues64(s2 / k - mean[:, :, None] * mean[:, None, :]).clamp(min=0)
        e = w / (w.sum(1, keepdim=True) + 1e-3)
        ent = -(e * torch.log(e + 1e-3)).sum(1)
        better = use & (ent < best)
        best, k_opt = torch.where(better, ent, best), torch.where(better, k, k_opt)
    del s1, s2
    out = torch.zeros((n, 12), dtype=torch.float64, device=DEVICE)
    place = torch.arange(width, device=DEVICE)
    for a in range(0, n, 1 << 18):
        at = (ptr[a:a + (1 << 18), None][:k_opt[a:a + (1 << 18)].shape[0]] + place).clamp(max=flat.shape[0] - 1)
        out[a:a + (1 << 18), :11] = _rows64(xyz, flat[at], k_opt[a:a + (1 << 18)])
    out[:, 11] = k_opt
    return out


def _eigenvalues64(c):
    """Eigenvalues of symmetric (n, 3, 3) matrices by the trigonometric closed form (ranking of candidate sizes)."""
    q = (c[:, 0, 0] + c[:, 1, 1] + c[:, 2, 2]) / 3
    b = c - q[:, None, None] * torch.eye(3, dtype=c.dtype, device=c.device)
    p = torch.sqrt((b * b).sum((1, 2)) / 6)
    safe = torch.where(p > 0, p, torch.ones_like(p))
    det = (b[:, 0, 0] * (b[:, 1, 1] * b[:, 2, 2] - b[:, 1, 2] ** 2) - b[:, 0, 1] * (b[:, 0, 1] * b[:, 2, 2] - b[:, 1, 2] * b[:, 0, 2])
           + b[:, 0, 2] * (b[:, 0, 1] * b[:, 1, 2] - b[:, 1, 1] * b[:, 0, 2]))
    phi = torch.acos((det / (2 * safe ** 3)).clamp(-1, 1)) / 3
    hi, lo = q + 2 * p * torch.cos(phi), q + 2 * p * torch.cos(phi + 2 * math.pi / 3)
    return torch.stack([lo, 3 * q - hi - lo, hi], 1)


def exact(case, seed):
    kind, k = case["kind"], case["k"]
    if kind in ("radius", "batch"):
        return None  # a brute-force search of millions of points takes too long
    if kind == "optimal":
        return _exact_optimal(case, seed)
    n = case["n"]
    if kind in ("features", "features_f64"):
        s = prepare(case, seed)
        nn = s["nn"].long().reshape(n, k)
        if s["scales"]:
            return torch.stack([_rows64(s["xyz"], nn, _full(n, min(v, k))) for v in s["scales"]], 1)
        return _rows64(s["xyz"], nn, _full(n, k))
    if float(n) * (case.get("m") or n) > PAIRS:
        return None
    if kind == "knn":
        data = _cloud(case, seed)
        query = _cloud(case, seed + 77_000, case["m"]) if case["m"] else data
        idx, _ = _search64(data, query, k)
        d2 = torch.cat([((data[idx[a:a + 65536]].double() - query[a:a + 65536, None].double()) ** 2).sum(2)
                        for a in range(0, query.shape[0], 65536)])
        return None, torch.sort(d2, dim=1).values
    if kind == "knn_features":
        xyz = _cloud(case, seed)
        idx, _ = _search64(xyz, xyz, k)
        scales = _scales(case)
        return torch.stack([_rows64(xyz, idx, _full(n, v)) for v in scales], 1) if scales else _rows64(xyz, idx, _full(n, k))
    xyz = _cloud(case, seed, dtype=getattr(torch, case["dtype"]))
    idx, hits = _search64(xyz, xyz, min(k, n), _radius(case))
    out = torch.zeros((n, len(case["ids"].split(","))), dtype=torch.float64, device=DEVICE)
    w, v = _pca64(xyz[idx].double(), torch.arange(idx.shape[1], device=DEVICE)[None, :] < hits[:, None])
    f = _features64(w, v)
    for j, name in enumerate(case["ids"].split(",")):
        column = {"Verticality": 1 - v[:, 2, 2].abs(), "Curvature": f[:, 10], "Planarity": f[:, 1], "Normal_z": v[:, 2, 2]}[name]
        out[:, j] = torch.where(hits >= 2, column, torch.zeros_like(column))
    return out.cpu().numpy() if case["host"] else out
