"""What this framework is timed on: closest-hit and shadow rays, distance queries and gradients.

Every case is a dict of plain values with a ``path`` (which entry point it calls) and that path's
sizes.  ``prepare`` makes the scene and the inputs from a seed, ``run`` is one pass through the
public API, ``work`` counts the bytes and operations the pass cannot do without, and ``exact``
gives what ``run`` returns as plain torch computes it in 64 bits, where that is feasible.
"""
import math

import numpy as np
import torch

import blazert_b200 as B
from blazert_b200 import autograd
from blazert_b200 import workloads as W

DBL_MAX = float(np.finfo(np.float64).max)
DEV = "cuda"
F64 = torch.float64
PAIR_BLOCK = 1 << 26     # (ray, primitive) pairs held at once by exact()
MAX_PAIRS = 1e11         # above this many pairs exact() would take too long: None


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one ray of a program that traces ray by ray, as the reference's examples do: a mouse
        # pick, a line-of-sight test; the latency of one call
        dict(name="single_ray", path="single", level=4),
        # one tile of a tiled renderer with host arrays (a few thousand rays, not a power of
        # two), a scene with every analytic kind
        dict(name="host_tile", path="host", mode="fp64", rays=3001, spheres=10_000,
             cylinders=1_000, planes=100),
        # a whole frame's worth of incoherent rays from ordinary numpy arrays, copies included
        dict(name="host_frame", path="host", mode="fp64", rays=1 << 20, spheres=10_000,
             cylinders=1_000, planes=100),
        # primary rays of a 512 x 512 image on the reference benchmark's sphere mesh, on the GPU
        dict(name="pinhole", path="pinhole", mode="fp64", level=4, width=512, height=512),
        # incoherent rays through spheres, planes and cylinders, on the GPU
        dict(name="primitives", path="primitives", mode="fp64", rays=1 << 20, spheres=10_000,
             cylinders=1_000, planes=100),
        # secondary (bounce) rays on a large terrain: the benchmark's default workload
        dict(name="terrain", path="terrain", mode="fp64", rays=1 << 23, grid=1024),
        # the same rays in the mixed mode
        dict(name="terrain_mixed", path="terrain", mode="mixed", rays=1 << 23, grid=1024),
        # shadow rays toward a light with a distance limit per ray, ragged sizes
        dict(name="terrain_shadow", path="shadow", mode="fp64", rays=1_000_003, grid=701),
        # many small scenes in one launch (a batch of objects), mixed mode
        dict(name="batch", path="batch", mode="mixed", scenes=48, rays=3_000_000),
        # a fitting step: closest hits, a loss on distances and normals, gradients of rays and
        # geometry
        dict(name="gradient", path="gradient", rays=1_000_003, level=5, split=2_000, spheres=500),
        # point-to-primitive distances (collision checks) on every kind
        dict(name="distance", path="distance", points=1 << 20, level=5, spheres=10_000,
             cylinders=1_000, planes=100),
        # nearest surface of a scene (signed-distance sampling, proximity)
        dict(name="nearest", path="nearest", points=1 << 20, level=6, split=10_000, spheres=500),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["single", "host", "pinhole", "pinhole", "primitives", "primitives",
                       "terrain", "terrain", "shadow", "batch", "gradient", "distance", "nearest"])
    mode = rng.choice(["fp64", "mixed"])
    analytic = dict(spheres=_log_int(rng, 100, 10_000), cylinders=_log_int(rng, 10, 1_000),
                    planes=_log_int(rng, 5, 100))
    if path == "single":
        return dict(path=path, level=rng.randint(2, 6))
    if path in ("host", "primitives"):
        return dict(path=path, mode=mode, rays=_log_int(rng, 500, 1 << 20), **analytic)
    if path == "pinhole":
        return dict(path=path, mode=mode, level=rng.randint(2, 7), width=_log_int(rng, 60, 1200),
                    height=_log_int(rng, 60, 800))
    if path in ("terrain", "shadow"):
        return dict(path=path, mode=mode, rays=_log_int(rng, 10_000, (1 << 23) - 1),
                    grid=_log_int(rng, 65, 1024))
    if path == "batch":
        return dict(path=path, mode=mode, scenes=rng.randint(5, 48),
                    rays=_log_int(rng, 50_000, 3_000_000))
    if path == "gradient":
        return dict(path=path, rays=_log_int(rng, 10_000, 1_000_000), level=rng.randint(3, 5),
                    split=_log_int(rng, 10, 1_000), spheres=_log_int(rng, 20, 500))
    if path == "distance":
        return dict(path=path, points=_log_int(rng, 2_000, 1 << 20), level=rng.randint(2, 5),
                    **analytic)
    return dict(path=path, points=_log_int(rng, 2_000, 1 << 20), level=rng.randint(3, 6),
                split=_log_int(rng, 10, 1_000), spheres=_log_int(rng, 20, 500))


# ------------------------------------------------------------------------------------ the inputs
def _scene(spec):
    s = B.Scene()
    for kind in spec.order:
        getattr(s, "add_" + kind)(*getattr(spec, kind).values())
    s.commit()
    return s


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _unit(x):
    return x / x.norm(dim=-1, keepdim=True)


def _analytic_spec(case, seed):
    return W.mixed_primitives(n_rays=1, n_spheres=case["spheres"], n_cylinders=case["cylinders"],
                              n_planes=case["planes"], seed=seed).scene


def _box_rays(g, n):
    """Incoherent rays: origins uniform in [-120, 120]^3, isotropic directions."""
    return 240.0 * _rand(g, n, 3) - 120.0, _unit(_randn(g, n, 3))


def _ball_rays(g, n, radius):
    """Rays from a sphere around the scene toward points of the unit ball."""
    o = radius * _unit(_randn(g, n, 3))
    q = _unit(_randn(g, n, 3)) * _rand(g, n, 1) ** (1.0 / 3.0)
    return o, _unit(q - o)


def _pinhole_rays(case, seed):
    """A pinhole camera at distance 3, turned about the y axis by an angle from the seed."""
    w, h = case["width"], case["height"]
    tan = math.tan(math.radians(30.0))
    i = (2.0 * (torch.arange(w, device=DEV, dtype=F64) + 0.5) / w - 1.0) * tan * (w / h)
    j = (1.0 - 2.0 * (torch.arange(h, device=DEV, dtype=F64) + 0.5) / h) * tan
    x = i[None, :].expand(h, w).reshape(-1)
    y = j[:, None].expand(h, w).reshape(-1)
    a = 0.37 * seed
    c, s = math.cos(a), math.sin(a)
    z = -torch.ones_like(x)
    d = _unit(torch.stack([c * x + s * z, y, c * z - s * x], 1))
    o = torch.tensor([3.0 * s, 0.0, 3.0 * c], device=DEV, dtype=F64).expand(w * h, 3).contiguous()
    return o, d.contiguous()


def _surface_points(g, verts, faces, n):
    """Points uniform on a terrain's surface (by area) and the upward unit normals there."""
    v0, v1, v2 = verts[faces[:, 0]], verts[faces[:, 1]], verts[faces[:, 2]]
    cr = torch.linalg.cross(v1 - v0, v2 - v0)
    area = cr.norm(dim=1)
    nf = cr / area[:, None] * torch.sign(cr[:, 2:3])
    cdf = torch.cumsum(area, 0)
    tri = torch.searchsorted(cdf, _rand(g, n) * cdf[-1]).clamp(max=len(area) - 1)
    r1, r2 = _rand(g, n, 1).sqrt(), _rand(g, n, 1)
    p = (1 - r1) * v0[tri] + r1 * (1 - r2) * v1[tri] + r1 * r2 * v2[tri]
    return p, nf[tri]


def _bounce_rays(g, verts, faces, n):
    """Secondary rays: cosine-weighted about the surface normal, offset by 1e-6 along it."""
    p, nrm = _surface_points(g, verts, faces, n)
    d = nrm + _unit(_randn(g, n, 3))  # cosine-weighted
    return p + 1e-6 * nrm, _unit(d)


def _light_rays(g, verts, faces, n):
    """Shadow rays toward one light above the terrain, and the distances to it."""
    p, nrm = _surface_points(g, verts, faces, n)
    light = torch.tensor([300.0, 650.0, 220.0], device=DEV, dtype=F64)
    o = p + 1e-6 * nrm
    d = light - o
    dist = d.norm(dim=1)
    return o, d / dist[:, None], dist


def _mesh_tensors(spec):
    v = torch.from_numpy(spec.mesh["vertices"]).to(DEV)
    f = torch.from_numpy(spec.mesh["faces"].astype(np.int64)).to(DEV)
    return v, f


def _terrain_spec(case, seed):
    return W.SceneSpec().add_mesh(*W.heightfield_mesh(case["grid"], seed=seed))


def _fitting_spec(case, seed):
    return W.adjoint_scene(n_rays=1, seed=seed, level=case["level"], n_split=case["split"],
                           n_spheres=case["spheres"]).scene


def _batch_specs(case, seed):
    """Scenes of different sizes (icospheres of levels 3 to 5, each stretched at random) and
    ray counts spread over two orders of magnitude that add up to case["rays"]."""
    rng = np.random.default_rng(seed)
    bases = {lv: W.icosphere(lv) for lv in (3, 4, 5)}
    specs = []
    for _ in range(case["scenes"]):
        v, f = bases[int(rng.integers(3, 6))]
        v = v * rng.uniform(0.8, 1.2, (1, 3)) + 0.03 * np.sin(v @ rng.uniform(2.0, 6.0, (3, 3)))
        specs.append(W.SceneSpec().add_mesh(v, f))
    share = np.exp(rng.uniform(0.0, math.log(100.0), case["scenes"]))
    cuts = np.floor(np.cumsum(share) / share.sum() * case["rays"]).astype(np.int64)
    cuts[-1] = case["rays"]
    return specs, [0] + [int(c) for c in cuts]


def _distance_spec(case, seed):
    spec = _analytic_spec(case, seed)
    return spec.add_mesh(*W.icosphere(case["level"]))


def _distance_queries(spec, case, g):
    """Per kind: random primitives and points around them at scales from 0.01 to 50."""
    n = case["points"]
    scales = torch.tensor([0.01, 0.3, 1.0, 5.0, 50.0], device=DEV, dtype=F64)
    out = {}
    for kind in spec.order:
        col = getattr(spec, kind)
        if kind == "mesh":
            v, f = _mesh_tensors(spec)
            centre = v[f].mean(1)
        else:
            centre = torch.from_numpy(col["centers"]).to(DEV)
        ids = torch.randint(0, len(centre), (n,), generator=g, device=DEV)
        sc = scales[torch.randint(0, 5, (n,), generator=g, device=DEV)]
        out[kind] = (ids.to(torch.int32), centre[ids] + sc[:, None] * _randn(g, n, 3))
    return out


def _inputs(case, seed):
    """(scene spec or specs, inputs) of a case, from the seed alone."""
    g = _gen(seed)
    path = case["path"]
    if path == "single":
        spec = W.SceneSpec().add_mesh(*W.icosphere(case["level"]))
        o, d = _ball_rays(g, 1, 3.0)
        return spec, (o, d)
    if path in ("host", "primitives"):
        return _analytic_spec(case, seed), _box_rays(g, case["rays"])
    if path == "pinhole":
        return W.SceneSpec().add_mesh(*W.icosphere(case["level"])), _pinhole_rays(case, seed)
    if path in ("terrain", "shadow"):
        spec = _terrain_spec(case, seed)
        make = _bounce_rays if path == "terrain" else _light_rays
        return spec, make(g, *_mesh_tensors(spec), case["rays"])
    if path == "batch":
        specs, offsets = _batch_specs(case, seed)
        return specs, (offsets, *_ball_rays(g, case["rays"], 3.0))
    if path == "gradient":
        spec = _fitting_spec(case, seed)
        n = case["rays"]
        return spec, (*_ball_rays(g, n, 4.0), _randn(g, n), _randn(g, n, 3))
    if path == "distance":
        spec = _distance_spec(case, seed)
        return spec, _distance_queries(spec, case, g)
    spec = _fitting_spec(case, seed)
    return spec, (5.0 * _rand(g, case["points"], 3) - 2.5,)


def prepare(case, seed):
    path = case["path"]
    spec, x = _inputs(case, seed)
    st = dict(path=path, mode=case.get("mode", "fp64"))
    if path == "batch":
        st["scenes"] = [_scene(s) for s in spec]
        st["batch"] = B.Batch(st["scenes"])
        st["offsets"], st["o"], st["d"] = x
        n = case["rays"]
        # a program that replays a batch keeps its result arrays
        st["out"] = dict(t=torch.empty(n, dtype=F64, device=DEV),
                         uv=torch.empty((n, 2), dtype=F64, device=DEV),
                         normal=torch.empty((n, 3), dtype=F64, device=DEV),
                         prim=torch.empty(n, dtype=torch.int32, device=DEV),
                         geom=torch.empty(n, dtype=torch.int32, device=DEV),
                         hit=torch.empty(n, dtype=torch.uint8, device=DEV))
        return st
    st["scene"] = _scene(spec)
    if path == "single":
        o, d = x[0].cpu().numpy()[0], x[1].cpu().numpy()[0]
        st["ray"] = B.Ray(o, d)
    elif path == "host":
        st["o"], st["d"] = x[0].cpu().numpy(), x[1].cpu().numpy()
    elif path == "shadow":
        st["o"], st["d"], st["tmax"] = x
    elif path == "gradient":
        st["o"], st["d"] = x[0].requires_grad_(), x[1].requires_grad_()
        st["wt"], st["wn"] = x[2], x[3]
        st["v"] = torch.from_numpy(spec.mesh["vertices"]).to(DEV).requires_grad_()
        st["c"] = torch.from_numpy(spec.spheres["centers"]).to(DEV).requires_grad_()
        st["r"] = torch.from_numpy(spec.spheres["radii"]).to(DEV).requires_grad_()
    elif path == "distance":
        st["queries"] = x
    elif path == "nearest":
        st["points"] = x[0]
    else:
        st["o"], st["d"] = x
    return st


# ------------------------------------------------------------------------------------- one pass
RESULT = ("t", "uv", "normal", "prim", "geom", "hit")


def run(st):
    path = st["path"]
    if path == "single":
        hit, rh = st["scene"].intersect1(st["ray"])
        return dict(t=np.array([rh.hit_distance]), uv=rh.uv[None], normal=rh.normal[None],
                    prim=np.array([rh.prim_id], np.uint32), geom=np.array([rh.geom_id], np.uint32),
                    hit=np.array([hit], np.uint8))
    if path == "batch":
        out = st["batch"].intersect(st["offsets"], st["o"], st["d"], out=st["out"],
                                    mode=st["mode"])
        return {k: out[k] for k in RESULT}
    if path == "gradient":
        t, uv, normal, prim, geom, hit = autograd.trace(st["scene"], st["o"], st["d"],
                                                        vertices=st["v"], centers=st["c"],
                                                        radii=st["r"])
        some = hit.bool()
        loss = (st["wt"] * torch.where(some, t, 0.0) ** 2).sum() + (st["wn"] * normal).sum()
        go, gd, gv, gc, gr = torch.autograd.grad(loss, [st["o"], st["d"], st["v"], st["c"],
                                                        st["r"]])
        return dict(t=t.detach(), uv=uv.detach(), normal=normal.detach(), prim=prim, geom=geom,
                    hit=hit, grad_origins=go, grad_directions=gd, grad_vertices=gv,
                    grad_centers=gc, grad_radii=gr)
    if path == "distance":
        out = {}
        for kind, (ids, pts) in st["queries"].items():
            r = st["scene"].distance_to_surface(kind, ids, pts, closest=kind == "mesh")
            if kind == "mesh":
                out[kind], out["closest"] = r
            else:
                out[kind] = r
        return out
    if path == "nearest":
        out = st["scene"].closest_surface(st["points"])
        return {k: out[k] for k in ("distance", "prim", "geom")}
    if path == "shadow":
        out = st["scene"].intersectN(st["o"], st["d"], tmax=st["tmax"], mode=st["mode"],
                                     any_hit=True)
    else:
        out = st["scene"].intersectN(st["o"], st["d"], mode=st["mode"])
    return {k: out[k] for k in RESULT}


# -------------------------------------------------------------------- what a pass cannot do without
RAY_IN, RAY_OUT = 48, 57  # origin and direction; t, uv, normal, prim, geom, hit
TRI_BYTES, SPHERE_BYTES, PLANE_BYTES, CYL_BYTES = 12 + 12, 32, 112, 120


def _tree_flops(prims):
    """Per query: both children of one node per level of a balanced tree over leaves of four
    (a slab test is 6 subtractions, 6 products and 6 comparisons), and one leaf's four tests."""
    levels = max(1.0, math.log2(max(2, prims) / 4.0))
    return levels * 2 * 18 + 4 * 60


def work(case):
    path = case["path"]
    geo = (case.get("spheres", 0) * SPHERE_BYTES + case.get("planes", 0) * PLANE_BYTES
           + case.get("cylinders", 0) * CYL_BYTES)
    tris = 20 * 4 ** case["level"] if "level" in case else 0
    if "grid" in case:
        tris = 2 * (case["grid"] - 1) ** 2
    geo += (tris + case.get("split", 0)) * TRI_BYTES
    kinds = [k for k in (tris, case.get("spheres", 0), case.get("planes", 0),
                         case.get("cylinders", 0)) if k]
    per_query = sum(_tree_flops(k) for k in kinds)
    if path == "single":  # one path through the tree, not the whole scene
        return {"bytes": RAY_IN + RAY_OUT + 64 * math.log2(tris), "flops": per_query}
    if path == "batch":
        tris = 20 * 4 ** 4
        return {"bytes": case["rays"] * (RAY_IN + RAY_OUT) + case["scenes"] * tris * TRI_BYTES,
                "flops": case["rays"] * _tree_flops(tris)}
    if path == "distance":
        n = case["points"]
        # ids and points in, distances out (closest points too for triangles); the ellipse
        # search of a cylinder converges in about six steps of 40 operations
        return {"bytes": geo + n * (4 * (4 + 24 + 8) + 24), "flops": n * (10 + 40 + 90 + 6 * 40)}
    if path == "nearest":
        n = case["points"]
        return {"bytes": geo + n * (24 + 8 + 4 + 4), "flops": n * per_query}
    n = case["rays"] if "rays" in case else case["width"] * case["height"]
    per_ray = RAY_IN + RAY_OUT + (8 if path == "shadow" else 0)
    if path == "gradient":
        # the loss and its gradients: dL/dt, dL/dn read, ray gradients written, geometry
        # gradients written once
        return {"bytes": n * (per_ray + 8 + 24 + 48) + geo + tris * 12 + case["spheres"] * 32,
                "flops": n * (per_query + 400)}
    return {"bytes": n * per_ray + geo, "flops": n * per_query}


# ------------------------------------------------------------------- the same in plain torch, 64 bits
def _dot(a, b):
    return (a * b).sum(-1)


def _vertex_normals(v, f):
    m = _unit(torch.linalg.cross(v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]])) / 3.0
    n = torch.zeros_like(v)
    for k in range(3):
        n = n.index_add(0, f[:, k], m)
    return n


def _first_triangle(v, f, o, d, tmax):
    """Index of the nearest triangle each ray hits before tmax, or -1 (all pairs)."""
    a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
    normal = torch.linalg.cross(b - a, c - a)
    plane = _dot(normal, a)
    # the side of each edge the ray passes on: d . (p x q) + (o x d) . (q - p)
    edges = [torch.cat([torch.linalg.cross(p, q), q - p], 1) for p, q in ((a, b), (b, c), (c, a))]
    line = torch.cat([d, torch.linalg.cross(o, d)], 1)
    out = torch.empty(len(o), dtype=torch.int64, device=DEV)
    step = max(1, PAIR_BLOCK // len(f))
    for i in range(0, len(o), step):
        s = slice(i, i + step)
        e0, e1, e2 = (line[s] @ e.T for e in edges)
        inside = ((e0 >= 0) & (e1 >= 0) & (e2 >= 0)) | ((e0 <= 0) & (e1 <= 0) & (e2 <= 0))
        t = (plane[None] - o[s] @ normal.T) / (d[s] @ normal.T)
        t = torch.where(inside & (t >= 0) & (t < tmax[s, None]), t, math.inf)
        best = t.min(1)
        out[s] = torch.where(torch.isfinite(best.values), best.indices, -1)
    return out


def _triangle_hit(v, vn, f, tri, o, d):
    """t, u, v and shading normal of rays on given triangles, differentiable."""
    p = f[tri]
    a, b, c = v[p[:, 0]], v[p[:, 1]], v[p[:, 2]]
    e1, e2, q = b - a, c - a, o - a
    h = torch.linalg.cross(d, e2)
    k = torch.linalg.cross(q, e1)
    det = _dot(e1, h)
    t, u, w = _dot(e2, k) / det, _dot(q, h) / det, _dot(d, k) / det
    n = (vn[p[:, 0]] * (1.0 - u - w)[:, None] + vn[p[:, 1]] * u[:, None]
         + vn[p[:, 2]] * w[:, None])
    return t, torch.stack([u, w], 1), _unit(n)


def _first_sphere(c, r, o, d, tmax):
    """Index of the nearest sphere each ray hits before tmax, or -1 (all pairs)."""
    out = torch.empty(len(o), dtype=torch.int64, device=DEV)
    step = max(1, PAIR_BLOCK // len(c))
    for i in range(0, len(o), step):
        s = slice(i, i + step)
        q = o[s, None] - c[None]
        half_b = (q * d[s, None]).sum(-1)
        disc = half_b ** 2 - ((q * q).sum(-1) - r ** 2)
        root = disc.clamp(min=0).sqrt()
        t = torch.where(-half_b - root > 0, -half_b - root, -half_b + root)
        t = torch.where((disc >= 0) & (t > 0) & (t < tmax[s, None]), t, math.inf)
        best = t.min(1)
        out[s] = torch.where(torch.isfinite(best.values), best.indices, -1)
    return out


def _sphere_hit(c, r, k, o, d):
    q = o - c[k]
    half_b = _dot(q, d)
    root = (half_b ** 2 - (_dot(q, q) - r[k] ** 2)).sqrt()
    t = torch.where(-half_b - root > 0, -half_b - root, -half_b + root)
    return t, _unit(o + t[:, None] * d - c[k])


def _exact_hits(spec, o, d, v=None, c=None, r=None):
    """t, uv, normal of the closest hits on a mesh and, with it, spheres; differentiable in
    the rays and in v, c, r."""
    f = torch.from_numpy(spec.mesh["faces"].astype(np.int64)).to(DEV)
    v = torch.from_numpy(spec.mesh["vertices"]).to(DEV) if v is None else v
    n = len(o)
    far = torch.full((n,), math.inf, device=DEV, dtype=F64)
    rd = _unit(d)
    with torch.no_grad():
        tri = _first_triangle(v, f, o, rd, far)
    hit_t = (tri >= 0).nonzero()[:, 0]
    t = torch.full((n,), DBL_MAX, device=DEV, dtype=F64)
    uv, normal = torch.zeros(n, 2, device=DEV, dtype=F64), torch.zeros(n, 3, device=DEV, dtype=F64)
    a, b, m = _triangle_hit(v, _vertex_normals(v, f), f, tri[hit_t], o[hit_t], rd[hit_t])
    t = t.index_put((hit_t,), a)
    uv = uv.index_put((hit_t,), b)
    normal = normal.index_put((hit_t,), m)
    if c is not None:
        with torch.no_grad():
            k = _first_sphere(c, r, o, rd, t)
        hit_s = (k >= 0).nonzero()[:, 0]
        a, m = _sphere_hit(c, r, k[hit_s], o[hit_s], rd[hit_s])
        t = t.index_put((hit_s,), a)
        uv = uv.index_put((hit_s,), torch.zeros(len(hit_s), 2, device=DEV, dtype=F64))
        normal = normal.index_put((hit_s,), m)
    return t, uv, normal


def _segment_point(a, b, p):
    e = b - a
    s = (_dot(p - a, e) / _dot(e, e)).clamp(0.0, 1.0)
    return a + s[..., None] * e


def _triangle_point(a, b, c, p):
    """Closest point of the triangle: its projection when inside, else on the nearest edge."""
    n = _unit(torch.linalg.cross((b - a).expand(p.shape), (c - a).expand(p.shape)))
    q = p - _dot(p - a, n)[..., None] * n
    side = [_dot(torch.linalg.cross((y - x).expand(q.shape), q - x), n)
            for x, y in ((a, b), (b, c), (c, a))]
    inside = (side[0] >= 0) & (side[1] >= 0) & (side[2] >= 0)
    best = _segment_point(a, b, p)
    for x, y in ((b, c), (c, a)):
        e = _segment_point(x, y, p)
        closer = (e - p).norm(dim=-1) < (best - p).norm(dim=-1)
        best = torch.where(closer[..., None], e, best)
    return torch.where(inside[..., None], q, best)


def _ellipse_distance(a, b, x, y):
    """Distance from (x, y) to the ellipse x^2/a^2 + y^2/b^2 = 1: bisection on the multiplier."""
    x, y = x.abs(), y.abs()
    swap = b > a
    a, b, x, y = (torch.where(swap, b, a), torch.where(swap, a, b), torch.where(swap, y, x),
                  torch.where(swap, x, y))
    # with z = multiplier / b^2 and k = (a / b)^2 the point is (k x / (z + k), y / (z + 1))
    k, ax, by = (a / b) ** 2, a / b * (x / b), y / b
    lo, hi = by - 1.0, torch.hypot(ax, by) - 1.0
    for _ in range(1100):
        mid = 0.5 * (lo + hi)
        if bool(((mid == lo) | (mid == hi)).all()):
            break
        val = (ax / (mid + k)) ** 2 + (by / (mid + 1.0)) ** 2 - 1.0
        lo, hi = torch.where(val > 0, mid, lo), torch.where(val > 0, hi, mid)
    z = 0.5 * (lo + hi)
    ex, ey = k * x / (z + k), y / (z + 1.0)
    return torch.hypot(ex - x, ey - y)


def _exact_distance(spec, queries):
    out = {}
    for kind, (ids, p) in queries.items():
        i = ids.long()
        col = {k: torch.from_numpy(x.astype(np.float64)).to(DEV)[i]
               for k, x in getattr(spec, kind).items()} if kind != "mesh" else None
        if kind == "mesh":
            v, f = _mesh_tensors(spec)
            t = v[f[i]]
            q = _triangle_point(t[:, 0], t[:, 1], t[:, 2], p)
            out["mesh"], out["closest"] = (q - p).norm(dim=1), q
        elif kind == "spheres":
            out[kind] = ((col["centers"] - p).norm(dim=1) - col["radii"]).abs()
        else:
            c = col["centers"]
            lp = torch.einsum("nij,ni->nj", col["rotations"], p - c)
            if kind == "planes":  # the reference compares the local point with the world centre
                dx, dy = col["dxs"] / 2, col["dys"] / 2
                on = ((lp[:, 0] - c[:, 0]).abs() <= dx) & ((lp[:, 1] - c[:, 1]).abs() <= dy)
                out[kind] = torch.where(on, lp[:, 2].abs(), DBL_MAX)
            else:
                a, b, h2 = col["semi_axes_a"], col["semi_axes_b"], col["heights"] / 2
                x, y, z = lp.unbind(1)
                shell = _ellipse_distance(a, b, x, y)
                top, bottom = (z - h2).abs(), (z + h2).abs()
                cap = torch.minimum(top, bottom)
                inside = (x / a) ** 2 + (y / b) ** 2 < 1.0
                between = z.abs() < h2
                out[kind] = torch.where(
                    inside, torch.where(between, torch.minimum(shell, cap),
                                        torch.where(z > 0, top, bottom)),
                    torch.where(between, shell, torch.hypot(shell, cap)))
    return out


def _exact_nearest(spec, p):
    """Distance to the nearest surface over all pairs."""
    v, f = _mesh_tensors(spec)
    t = v[f]
    c = torch.from_numpy(spec.spheres["centers"]).to(DEV)
    r = torch.from_numpy(spec.spheres["radii"]).to(DEV)
    out = torch.empty(len(p), device=DEV, dtype=F64)
    step = max(1, (PAIR_BLOCK >> 3) // len(f))
    for i in range(0, len(p), step):
        q = p[i:i + step, None]
        best = (_triangle_point(t[None, :, 0], t[None, :, 1], t[None, :, 2],
                                q.expand(-1, len(f), 3)) - q).norm(dim=-1).min(1).values
        sph = ((c[None] - q).norm(dim=-1) - r).abs().min(1).values
        out[i:i + step] = torch.minimum(best, sph)
    return out


def exact(case, seed):
    """What run returns, in 64 bits by plain torch (ids and flags: None).  None for scenes with
    cylinders (the reference's cylinder test keeps the last hit, not the closest, so its results
    follow from its own tree order) and where all pairs would take too long."""
    path = case["path"]
    tris = 20 * 4 ** case["level"] + case.get("split", 0) if "level" in case else 0
    if "grid" in case:
        tris = 2 * (case["grid"] - 1) ** 2
    queries = case.get("rays", case.get("points", case.get("width", 1) * case.get("height", 1)))
    if path in ("host", "primitives", "batch", "shadow"):
        return None  # cylinders; many scenes; any hit, whichever comes first
    if path != "distance" and tris * queries > (MAX_PAIRS / 20 if path == "nearest" else MAX_PAIRS):
        return None
    spec, x = _inputs(case, seed)
    if path == "distance":
        return _exact_distance(spec, x)
    ids = dict(prim=None, geom=None, hit=None)
    if path == "nearest":
        return dict(distance=_exact_nearest(spec, x[0]), prim=None, geom=None)
    if path == "gradient":
        o, d = x[0].requires_grad_(), x[1].requires_grad_()
        v = torch.from_numpy(spec.mesh["vertices"]).to(DEV).requires_grad_()
        c = torch.from_numpy(spec.spheres["centers"]).to(DEV).requires_grad_()
        r = torch.from_numpy(spec.spheres["radii"]).to(DEV).requires_grad_()
        t, uv, normal = _exact_hits(spec, o, d, v, c, r)
        some = t < DBL_MAX
        loss = (x[2] * torch.where(some, t, 0.0) ** 2).sum() + (x[3] * normal).sum()
        g = torch.autograd.grad(loss, [o, d, v, c, r])
        return dict(t=t.detach(), uv=uv.detach(), normal=normal.detach(), **ids,
                    grad_origins=g[0], grad_directions=g[1], grad_vertices=g[2],
                    grad_centers=g[3], grad_radii=g[4])
    t, uv, normal = _exact_hits(spec, x[0], x[1])
    return dict(t=t, uv=uv, normal=normal, **ids)
