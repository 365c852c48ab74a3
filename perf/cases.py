"""Performance cases of the spatial-query path: the calls that programs using this framework make, through its public
Python entry points, from the smallest ones (latency) to the largest.

``listed()`` gives the fixed cases and ``draw(rng)`` one more of the same ranges; ``prepare`` makes what a program has in
hand before the call (inputs on the GPU, the BVH it keeps), ``run`` makes one call and returns its outputs, ``work`` counts
the bytes and operations that no implementation can do without, and ``exact`` gives the outputs from plain 64-bit
arithmetic (brute force) where that takes seconds.

Sizes are those of the benchmark's configurations and of the tests, with odd ones among them.
"""

import math

import numpy as np
import torch

from thea_gb300 import bvh as B
from thea_gb300 import workloads as W

# Brute-force pair counts up to which exact() answers (a few seconds each on the GPU)
CLOSEST_PAIRS = 4 << 30
RAY_PAIRS = 4 << 30
KNN_PAIRS = 16 << 30
RADIUS_PAIRS = 48 << 30


def listed():
    return [
        # One ICP step of a registration loop: a small scan against a small mesh, points near the surface. Latency.
        {"name": "closest_icp", "kind": "closest", "level": 4, "n": 1000, "near": True, "precision": "fp32"},
        # Signed-distance-like sampling around a mesh: the benchmark's plain closest-point configuration, full size.
        {"name": "closest_box", "kind": "closest", "level": 6, "n": 262144, "near": False, "precision": "fp32"},
        # The same with the FP64 re-check (exact element choice near edges), at an odd size.
        {"name": "closest_fp64", "kind": "closest", "level": 5, "n": 100003, "near": False, "precision": "fp64"},
        # A sensor sweep or picking: a thousand rays with normals against a small terrain. Latency.
        {"name": "ray_probe", "kind": "ray", "grid": 129, "n": 1000, "normals": True},
        # The benchmark's headline: first hits of 4 M rays on a 2 M-triangle terrain.
        {"name": "ray_terrain", "kind": "ray", "grid": 1024, "n": 4194304, "normals": False},
        # Feature transfer between point sets: the k nearest points of scattered queries.
        {"name": "knn_points", "kind": "knn", "points": 262144, "n": 50021, "k": 8},
        # The benchmark's k-nearest-neighbour graph of surface samples, full size.
        {"name": "knn_graph", "kind": "knn_self", "points": 1048576, "k": 16},
        # Many meshes of uneven size in one call: a sixteenth of the benchmark's batched configuration.
        {"name": "forest_closest", "kind": "forest", "meshes": 256, "min_level": 2, "max_level": 7, "min_q": 1000,
         "max_q": 100000, "precision": "fp32"},
        # A deforming mesh: the BVH is rebuilt every frame, then queried.
        {"name": "rebuild_closest", "kind": "rebuild", "level": 6, "n": 16384},
        # Every point within a radius of every sample (density, normals, outlier filters), CSR with distances.
        {"name": "radius_points", "kind": "radius", "points": 200003, "mean": 24},
        # The sample proximity graph of a surface with reachability against its mesh.
        {"name": "sample_graph", "kind": "graph", "level": 6, "points": 262144, "degree": 8},
        # Area-weighted surface sampling with the reference's generator: the samples of the k-NN graph.
        {"name": "sample_area", "kind": "sample", "level": 6, "n": 1048576},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "closest", "ray", "ray", "knn", "knn_self", "forest", "rebuild", "radius", "graph",
                       "sample"])
    if kind == "closest":
        return {"kind": kind, "level": rng.randint(3, 6), "n": _log_int(rng, 1000, 262144),
                "near": rng.random() < 0.5, "precision": rng.choice(["fp32", "fp32", "fp64"])}
    if kind == "ray":
        return {"kind": kind, "grid": _log_int(rng, 65, 1024), "n": _log_int(rng, 1000, 4194304),
                "normals": rng.random() < 0.5}
    if kind == "knn":
        return {"kind": kind, "points": _log_int(rng, 4096, 1048576), "n": _log_int(rng, 1000, 262144),
                "k": rng.choice([1, 3, 4, 8, 10, 16])}
    if kind == "knn_self":
        return {"kind": kind, "points": _log_int(rng, 4096, 1048576), "k": rng.choice([4, 8, 12, 16])}
    if kind == "forest":
        return {"kind": kind, "meshes": _log_int(rng, 8, 256), "min_level": 2, "max_level": rng.randint(4, 6),
                "min_q": 1000, "max_q": _log_int(rng, 4000, 50000), "precision": rng.choice(["fp32", "fp64"])}
    if kind == "rebuild":
        return {"kind": kind, "level": rng.randint(3, 6), "n": _log_int(rng, 1000, 65536)}
    if kind == "radius":
        return {"kind": kind, "points": _log_int(rng, 4096, 262144), "mean": rng.randint(6, 32)}
    if kind == "graph":
        return {"kind": kind, "level": rng.randint(4, 6), "points": _log_int(rng, 8192, 262144),
                "degree": rng.choice([6, 8, 12])}
    return {"kind": kind, "level": rng.randint(3, 6), "n": _log_int(rng, 4096, 1048576)}


# ---------------------------------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")


def _sphere_mesh(level, seed):
    v, f = W.noisy_icosphere(level, int(seed))
    return torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()


def _mesh_samples(g, v, f, n):
    """n points uniform by area on the mesh with their face normals."""
    v0, v1, v2 = (v[f[:, i].long()] for i in range(3))
    c = torch.linalg.cross(v1 - v0, v2 - v0)
    cdf = torch.cumsum(c.double().norm(dim=1), 0)
    face = torch.searchsorted(cdf, torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cdf[-1])
    face = face.clamp(max=len(f) - 1)
    s, t = torch.rand((2, n, 1), generator=g, device="cuda")
    over = s + t > 1
    s, t = torch.where(over, 1 - s, s), torch.where(over, 1 - t, t)
    p = v0[face] + s * (v1 - v0)[face] + t * (v2 - v0)[face]
    return p.contiguous(), torch.nn.functional.normalize(c[face], dim=1).contiguous()


def _sphere_points(g, n):
    d = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    return (d * (1.0 + 0.01 * torch.randn((n, 1), generator=g, device="cuda"))).contiguous()


def _terrain(n, g):
    """n x n vertices over [0,1]^2 with fBm value-noise heights, two triangles per cell."""
    u = torch.linspace(0, 1, n, device="cuda")
    x, y = torch.meshgrid(u, u, indexing="ij")
    z = torch.zeros_like(x)
    amp, freq = 0.1, 4
    for _ in range(6):
        lat = torch.rand((freq + 1, freq + 1), generator=g, device="cuda")
        ix, iy = ((c * freq).floor().long().clamp(max=freq - 1) for c in (x, y))
        tx, ty = x * freq - ix, y * freq - iy
        sx, sy = tx * tx * (3 - 2 * tx), ty * ty * (3 - 2 * ty)
        a = lat[ix, iy] + (lat[ix + 1, iy] - lat[ix, iy]) * sx
        b = lat[ix, iy + 1] + (lat[ix + 1, iy + 1] - lat[ix, iy + 1]) * sx
        z += amp * ((a + (b - a) * sy) * 2 - 1)
        amp, freq = amp * 0.5, freq * 2
    v = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1).contiguous()
    i = torch.arange(n - 1, device="cuda")
    v00 = (i[:, None] * n + i[None]).reshape(-1)
    f = torch.stack([torch.stack([v00, v00 + n, v00 + n + 1], 1), torch.stack([v00, v00 + n + 1, v00 + 1], 1)], 1)
    return v, f.reshape(-1, 3).to(torch.int32).contiguous()


def _rays_down(g, n):
    o = torch.rand((n, 3), generator=g, device="cuda")
    o[:, 2] = 0.5
    u, w = torch.rand((2, n), generator=g, device="cuda")
    r, phi = u.sqrt(), 2 * math.pi * w
    d = torch.stack([r * phi.cos(), r * phi.sin(), -(1 - u).clamp(min=0).sqrt()], 1)
    return o, d.contiguous()


def _forest_sizes(case):
    """Subdivision level and query count of each mesh: levels uniform, query counts log-uniform. They belong to the case."""
    levels, _, nq, _ = W.config3_spec(case["meshes"], seed=case["meshes"], min_level=case["min_level"],
                                      max_level=case["max_level"], min_q=case["min_q"], max_q=case["max_q"])
    return levels, nq


def _forest(case, g):
    """Noisy spheres stretched per axis by 0.5 to 2, each with queries uniform in its box grown by half."""
    levels, nq = _forest_sizes(case)
    v_all, f_all, q_all, base = [], [], [], 0
    for level, n in zip(levels, nq):
        v, f = W.icosphere(int(level))
        v = torch.from_numpy(v).float().cuda()
        v = v * (1 + 0.01 * torch.randn((len(v), 1), generator=g, device="cuda")) * _uniform(g, 1, 0.5, 2.0)
        lo, hi = v.min(0).values, v.max(0).values
        q_all.append((lo + hi) / 2 + 1.5 * (hi - lo) * _uniform(g, int(n), -0.5, 0.5))
        v_all.append(v)
        f_all.append((torch.from_numpy(f).cuda() + base).to(torch.int32))
        base += len(v)
    foff = np.cumsum([0] + [len(f) for f in f_all]).astype(np.int64)
    qoff = torch.from_numpy(np.cumsum([0] + [len(q) for q in q_all]).astype(np.int64)).cuda()
    return {"v": torch.cat(v_all), "f": torch.cat(f_all), "foff": foff, "q": torch.cat(q_all), "qoff": qoff}


def _inputs(case, seed):
    """The case's inputs (CUDA tensors and plain values), from the seed alone."""
    kind = case["kind"]
    g = _generator(seed)
    if kind in ("closest", "rebuild"):
        v, f = _sphere_mesh(case["level"], seed)
        if case.get("near"):
            p, _ = _mesh_samples(g, v, f, case["n"])
            q = p + 0.02 * torch.randn(p.shape, generator=g, device="cuda")
        else:
            q = _uniform(g, case["n"], -1.5, 1.5)
        return {"v": v, "f": f, "q": q.contiguous()}
    if kind == "ray":
        v, f = _terrain(case["grid"], g)
        o, d = _rays_down(g, case["n"])
        return {"v": v, "f": f, "o": o, "d": d}
    if kind in ("knn", "knn_self"):
        out = {"p": _sphere_points(g, case["points"])}
        if kind == "knn":
            out["q"] = _sphere_points(g, case["n"])
        return out
    if kind == "forest":
        return _forest(case, g)
    if kind == "radius":
        # one set of points, mirrored and renumbered by the seed: the neighbours are others, their number is not
        n = case["points"]
        p = _sphere_points(_generator(n), n)[torch.randperm(n, generator=g, device="cuda")]
        sign = torch.where(torch.rand(3, generator=g, device="cuda") < 0.5, -1.0, 1.0)
        return {"p": (p * sign).contiguous(), "r": 2.0 * math.sqrt(case["mean"] / n),
                "self": torch.arange(n, dtype=torch.int32, device="cuda")}
    if kind == "graph":
        v, f = _sphere_mesh(case["level"], seed)
        p, nrm = _mesh_samples(g, v, f, case["points"])
        return {"v": v, "f": f, "p": p, "nrm": nrm, "seed": int(seed) & 0xffff}
    v, f = _sphere_mesh(case["level"], seed)
    return {"v": v, "f": f, "seed": int(seed) & 0xffff}


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind in ("closest", "ray"):
        s["bvh"] = B.MeshBvh(s["v"], s["f"])
    elif kind in ("knn", "knn_self", "radius"):
        s["bvh"] = B.PointBvh(s["p"])
    elif kind == "forest":
        s["bvh"] = B.MeshForest(s["v"], s["f"], s["foff"])
    elif kind == "graph":
        s["bvh"] = B.MeshBvh(s["v"], s["f"])
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "closest":
        if case["precision"] == "fp32":
            return state["bvh"].closest_element(state["q"])
        return state["bvh"].closest_element_ex(state["q"], precision="fp64", errors=False)[:3]
    if kind == "ray":
        t, idx, nrm = state["bvh"].ray_structure_intersection(state["o"], state["d"], normals=case["normals"])
        return (t, idx, nrm) if case["normals"] else (t, idx)
    if kind == "knn":
        return state["bvh"].k_closest_pairs(state["q"], case["k"])
    if kind == "knn_self":
        return state["bvh"].k_closest_self(case["k"], device=True)
    if kind == "forest":
        return state["bvh"].batch_closest_element(state["q"], state["qoff"], precision=case["precision"])[:2]
    if kind == "rebuild":
        bvh = B.MeshBvh(state["v"], state["f"])
        return bvh.closest_element(state["q"])
    if kind == "radius":
        return state["bvh"].radius_neighbors(state["p"], state["r"], exclude=state["self"])
    if kind == "graph":
        nbr, sep, deg, mean = B.sample_graph(state["p"], state["nrm"], max_degree=case["degree"], seed=state["seed"],
                                             surface=state["bvh"])
        return nbr, sep, deg, mean[0], mean[1]
    return B.sample_evenly_by_area(state["v"], state["f"], case["n"], state["seed"])


# ---------------------------------------------------------------------------------------------------------------------
# What one pass cannot do without: inputs read once, outputs written once, one element test per result
# ---------------------------------------------------------------------------------------------------------------------

def _sphere_bytes(level):
    faces = 20 * 4 ** level
    return 12 * faces + 12 * (faces // 2 + 2)


def work(case):
    kind = case["kind"]
    if kind == "closest":
        return {"bytes": 32 * case["n"] + _sphere_bytes(case["level"]), "flops": 100 * case["n"]}
    if kind == "rebuild":
        return {"bytes": 32 * case["n"] + _sphere_bytes(case["level"]),
                "flops": 100 * case["n"] + 50 * 20 * 4 ** case["level"]}
    if kind == "ray":
        g = case["grid"]
        return {"bytes": (44 if case["normals"] else 32) * case["n"] + 12 * g * g + 24 * (g - 1) ** 2,
                "flops": 60 * case["n"]}
    if kind == "knn":
        return {"bytes": 12 * case["points"] + (12 + 8 * case["k"]) * case["n"], "flops": 8 * case["k"] * case["n"]}
    if kind == "knn_self":
        return {"bytes": (12 + 8 * case["k"]) * case["points"], "flops": 8 * case["k"] * case["points"]}
    if kind == "forest":
        levels, nq = _forest_sizes(case)
        return {"bytes": 20 * int(nq.sum()) + sum(_sphere_bytes(int(x)) for x in levels),
                "flops": 100 * int(nq.sum())}
    if kind == "radius":
        n, m = case["points"], case["mean"]
        return {"bytes": (12 + 4 + 8 + 8 * m) * n, "flops": 8 * m * n}
    if kind == "graph":
        n, d = case["points"], case["degree"]
        return {"bytes": (24 + 4 + 8 * d) * n + _sphere_bytes(case["level"]), "flops": 20 * d * n}
    return {"bytes": 28 * case["n"] + _sphere_bytes(case["level"]), "flops": 30 * case["n"]}


# ---------------------------------------------------------------------------------------------------------------------
# Outputs from 64-bit arithmetic
# ---------------------------------------------------------------------------------------------------------------------

def _dot(a, b):
    return (a * b).sum(-1)


def _closest_point(q, a, b, c):
    """Closest point of the triangles (a, b, c) to the points q (broadcast, float64): the plane projection where it lies
    inside, else the nearest point of the three edges."""
    n = torch.linalg.cross(b - a, c - a, dim=-1)
    nn = _dot(n, n)
    proj = q - (_dot(q - a, n) / nn)[..., None] * n
    inside = torch.ones(proj.shape[:-1], dtype=torch.bool, device=q.device)
    best, best_d = None, None
    for u, w in ((a, b), (b, c), (c, a)):
        e = w - u
        inside &= _dot(torch.linalg.cross(e.expand_as(proj), proj - u, dim=-1), n.expand_as(proj)) >= 0
        t = (_dot(q - u, e) / _dot(e, e)).clamp(0, 1)
        p = u + t[..., None] * e
        d = _dot(p - q, p - q)
        if best is None:
            best, best_d = p, d
        else:
            nearer = d < best_d
            best, best_d = torch.where(nearer[..., None], p, best), torch.minimum(d, best_d)
    cp = torch.where(inside[..., None], proj, best)
    return cp, _dot(cp - q, cp - q)


def _exact_closest(v, f, q):
    """Distances and closest points of q (float64): each point's candidates are the triangles whose centroid is within
    the reach of the nearest one, their vertices at most `reach` from it."""
    v, q = v.double(), q.double()
    a, b, c = (v[f[:, i].long()] for i in range(3))
    ctr = (a + b + c) / 3
    reach = torch.stack([(x - ctr).norm(dim=1) for x in (a, b, c)]).max()
    dist = torch.empty(len(q), dtype=torch.float64, device="cuda")
    cp = torch.empty((len(q), 3), dtype=torch.float64, device="cuda")
    step = max(1, (64 << 20) // len(f))
    for i in range(0, len(q), step):
        p = q[i:i + step]
        dc = torch.zeros((len(p), len(f)), dtype=torch.float64, device="cuda")
        for x in range(3):
            dc += (p[:, x, None] - ctr[None, :, x]) ** 2
        lim = dc.min(1).values.sqrt() + reach * (1 + 1e-9)
        row, tri = (dc <= (lim * lim)[:, None]).nonzero(as_tuple=True)
        pts, d2 = _closest_point(p[row], a[tri], b[tri], c[tri])
        best = torch.full((len(p),), math.inf, dtype=torch.float64, device="cuda").scatter_reduce(
            0, row, d2, reduce="amin")
        win = d2 == best[row]
        cp[i + row[win]] = pts[win]
        dist[i:i + step] = best.sqrt()
    return dist, cp


def _exact_rays(v, f, o, d):
    """First hit times (-1 on a miss) and unit face normals (zero on a miss), float64."""
    v, o, d = v.double(), o.double(), d.double()
    a, b, c = (v[f[:, i].long()] for i in range(3))
    e1, e2 = b - a, c - a
    n = torch.linalg.cross(e1, e2)
    t_out = torch.full((len(o),), -1.0, dtype=torch.float64, device="cuda")
    n_out = torch.zeros((len(o), 3), dtype=torch.float64, device="cuda")
    step = max(1, (4 << 20) // len(f))
    for i in range(0, len(o), step):
        oo, dd = o[i:i + step, None], d[i:i + step, None]
        s = oo - a
        dn = _dot(dd, n)
        m = torch.linalg.cross(s, dd.expand_as(s), dim=-1)
        t = -_dot(s, n) / dn
        u = -_dot(m, e2) / dn
        w = _dot(m, e1) / dn
        ok = (dn.abs() > 2.0 ** -23) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 0)
        t = torch.where(ok, t, math.inf)
        best, k = t.min(1)
        hit = best < math.inf
        t_out[i:i + step] = torch.where(hit, best, -1.0)
        n_out[i:i + step] = torch.where(hit[:, None], torch.nn.functional.normalize(n[k], dim=1), 0.0)
    return t_out, n_out


def _pair_d2(p, x, dtype):
    s = None
    for ax in (2, 1, 0):
        e = (x[None, :, ax].to(dtype) - p[:, ax, None].to(dtype)) ** 2
        s = e if s is None else e + s
    return s


def _exact_knn(p, q, k, skip_self):
    """Squared distances of the k nearest points, ascending, float64 (-1 past the number of points)."""
    out = torch.full((len(q), k), -1.0, dtype=torch.float64, device="cuda")
    m = min(k, len(p) - (1 if skip_self else 0))
    step = max(1, (256 << 20) // len(p))
    for i in range(0, len(q), step):
        d2 = _pair_d2(q[i:i + step], p, torch.float64)
        if skip_self:
            r = torch.arange(len(d2), device="cuda")
            d2[r, i + r] = math.inf
        out[i:i + step, :m] = torch.topk(d2, m, largest=False).values.sort(1).values
    return out


def _exact_radius(p, r):
    """Squared distances of the neighbours in CSR order, float64. Which points are neighbours is the FP32 comparison
    |x - p|^2 <= r * r that the entry point documents."""
    r2 = torch.tensor(r, dtype=torch.float32, device="cuda")
    r2 = r2 * r2
    parts = []
    step = max(1, (256 << 20) // len(p))
    for i in range(0, len(p), step):
        near = _pair_d2(p[i:i + step], p, torch.float32) <= r2
        k = torch.arange(len(near), device="cuda")
        near[k, i + k] = False
        row, col = near.nonzero(as_tuple=True)
        parts.append(((p[col].double() - p[i + row].double()) ** 2).sum(1))
    return torch.cat(parts)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("closest", "rebuild"):
        if case["n"] * 20 * 4 ** case["level"] > CLOSEST_PAIRS:
            return None
        s = _inputs(case, seed)
        dist, cp = _exact_closest(s["v"], s["f"], s["q"])
        return None, dist, cp
    if kind == "ray":
        if case["n"] * 2 * (case["grid"] - 1) ** 2 > RAY_PAIRS:
            return None
        s = _inputs(case, seed)
        t, nrm = _exact_rays(s["v"], s["f"], s["o"], s["d"])
        return (t, None, nrm) if case["normals"] else (t, None)
    if kind in ("knn", "knn_self"):
        n = case["n"] if kind == "knn" else case["points"]
        if n * case["points"] > KNN_PAIRS:
            return None
        s = _inputs(case, seed)
        return None, _exact_knn(s["p"], s["q"] if kind == "knn" else s["p"], case["k"], kind == "knn_self")
    if kind == "forest":
        levels, nq = _forest_sizes(case)
        if int((nq * 20 * 4 ** levels.astype(np.int64)).sum()) > CLOSEST_PAIRS:
            return None
        s = _inputs(case, seed)
        qoff = s["qoff"].tolist()
        dist = [_exact_closest(s["v"], s["f"][int(s["foff"][m]):int(s["foff"][m + 1])], s["q"][qoff[m]:qoff[m + 1]])[0]
                for m in range(case["meshes"])]
        return None, torch.cat(dist)
    if kind == "radius":
        if case["points"] ** 2 > RADIUS_PAIRS:
            return None
        s = _inputs(case, seed)
        return None, None, _exact_radius(s["p"], s["r"])
    return None
