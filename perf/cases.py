"""Performance cases of the acceleration-structure and participating-media path.

Each case is one pass of work that a program gives this framework through its
Python entry points.  Kinds:

  trace      closest hits of a batch of rays over a built single-scene handle
  shadow     any hit (occlusion) with a segment length per ray
  batch      closest hits over a batched handle with the tuned trace options
  frame      rebuild over moved vertices, then one closest-hit trace
  gradient   closest hits and their adjoint with respect to the vertices
  volume     ratio-tracking transmittance with checkpoints, and its adjoint
  scatter    delta tracking through a sparse brick grid
  render     the wavefront path tracer, with or without a medium

Geometry is either a random triangle soup in the unit cube (centroids
U[0,1]^3, vertices within +-half of the centroid) or an indexed, displaced
icosphere.  All inputs are made on the GPU from the seed.
"""
import functools
import math

import torch

import fledge_gb300 as F
from fledge_gb300 import scenes

DEVICE = "cuda:0"


@functools.lru_cache(maxsize=None)
def context():
    """The program's one context, on torch's stream."""
    return F.Context(0)


def listed():
    return [
        # A single interactive query: a small mesh, a few hundred rays.  Launches and host work.
        {"name": "trace_pick", "kind": "trace", "geometry": "sphere", "level": 3, "rays": "camera", "n_rays": 255},
        # The 65,536-triangle scene with 1,048,576 scattered rays, default options.
        {"name": "trace_soup_64k", "kind": "trace", "geometry": "soup", "n_tri": 65536, "rays": "scatter",
         "n_rays": 1 << 20},
        # Camera rays of a preview image on a surface mesh, default options.
        {"name": "trace_camera_330k", "kind": "trace", "geometry": "sphere", "level": 7, "rays": "camera",
         "n_rays": 1280 * 720},
        # Shadow rays from a surface to a light, any hit, an odd number of them.
        {"name": "shadow_330k", "kind": "shadow", "geometry": "sphere", "level": 7, "n_rays": 1999999},
        # Many scenes in one handle, 64 rays per triangle, the tuned layout and kernel options.
        {"name": "batch_24_scenes", "kind": "batch", "n_scenes": 24, "low": 1000, "high": 100000, "rays_per_tri": 64,
         "leaf": 3, "build_each": False},
        # A small dynamic scene: rebuilt every frame, few rays.  Latency of the build's stages.
        {"name": "frame_20k", "kind": "frame", "geometry": "soup", "n_tri": 20001, "n_rays": 4096},
        # A large dynamic scene: the build at the size where it is bound by memory.
        {"name": "frame_4m", "kind": "frame", "geometry": "soup", "n_tri": 4000003, "n_rays": 1 << 20},
        # A batch of scenes rebuilt in one segmented pass and traced with one ray per triangle.
        {"name": "frame_100_scenes", "kind": "batch", "n_scenes": 100, "low": 1000, "high": 100000, "rays_per_tri": 1,
         "leaf": 3, "build_each": True},
        # Vertex gradients of closest hits: the inner step of a fit to depth measurements.
        {"name": "gradient_50k", "kind": "gradient", "geometry": "soup", "n_tri": 50000, "n_rays": 500000},
        # Transmittance through the 256^3 grid and its gradient.
        {"name": "volume_256", "kind": "volume", "res": 256, "n_rays": 1 << 20},
        # Free-flight sampling through a mostly empty sparse grid.
        {"name": "scatter_sparse_192", "kind": "scatter", "res": 192, "n_rays": 1 << 21},
        # A whole image by the path tracer, the options its benchmark uses.
        {"name": "render_640x360", "kind": "render", "level": 6, "width": 640, "height": 360, "spp": 4,
         "max_depth": 5, "medium": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "shadow", "batch", "frame", "frame", "gradient", "volume", "scatter", "render"])
    if kind == "trace":
        if rng.random() < 0.5:
            return {"kind": kind, "geometry": "soup", "n_tri": _log_int(rng, 200, 300000),
                    "rays": rng.choice(["scatter", "camera"]), "n_rays": _log_int(rng, 200, 1 << 21)}
        return {"kind": kind, "geometry": "sphere", "level": rng.randint(2, 7), "rays": rng.choice(["scatter", "camera"]),
                "n_rays": _log_int(rng, 200, 1 << 21)}
    if kind == "shadow":
        if rng.random() < 0.5:
            return {"kind": kind, "geometry": "soup", "n_tri": _log_int(rng, 200, 300000),
                    "n_rays": _log_int(rng, 200, 1 << 21)}
        return {"kind": kind, "geometry": "sphere", "level": rng.randint(2, 7), "n_rays": _log_int(rng, 200, 1 << 21)}
    if kind == "batch":
        return {"kind": kind, "n_scenes": rng.randint(2, 100), "low": 1000, "high": _log_int(rng, 3000, 30000),
                "rays_per_tri": rng.choice([1, 4, 16]), "leaf": rng.randint(1, 4), "build_each": rng.random() < 0.5}
    if kind == "frame":
        return {"kind": kind, "geometry": "soup", "n_tri": _log_int(rng, 500, 3000000),
                "n_rays": _log_int(rng, 200, 1 << 20)}
    if kind == "gradient":
        return {"kind": kind, "geometry": "soup", "n_tri": _log_int(rng, 1000, 200000),
                "n_rays": _log_int(rng, 1000, 1 << 20)}
    if kind == "volume":
        return {"kind": kind, "res": _log_int(rng, 24, 256), "n_rays": _log_int(rng, 1000, 1 << 20)}
    if kind == "scatter":
        return {"kind": kind, "res": _log_int(rng, 24, 192), "n_rays": _log_int(rng, 1000, 1 << 21)}
    w = rng.randint(100, 640)
    return {"kind": kind, "level": rng.randint(4, 6), "width": w, "height": max(40, w * 9 // 16), "spp": rng.randint(1, 4),
            "max_depth": rng.randint(1, 5), "medium": rng.random() < 0.5}


# --------------------------------- inputs ----------------------------------

@functools.lru_cache(maxsize=2)
def _sphere(level):
    v, f = scenes.icosphere(level, amplitude=0.0)
    return torch.from_numpy(v), torch.from_numpy(f)


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, device=DEVICE, generator=g)


def _soup(n, g):
    # the benchmark's triangles up to its 65,536-triangle scene; above that the half size follows the spacing
    half = min(0.01, 0.4 * n ** (-1.0 / 3.0))
    cent = _rand(g, n, 1, 3)
    return (cent + (2.0 * _rand(g, n, 3, 3) - 1.0) * half).reshape(-1, 3).contiguous()


def _sphere_mesh(level, g):
    """Unit icosphere displaced by a few seeded waves (amplitude 0.05)."""
    v, f = _sphere(level)
    v = v.to(DEVICE)
    k = (_rand(g, 6, 3) - 0.5) * 24.0
    ph = _rand(g, 6) * 6.2831853
    r = 1.0 + 0.05 / 6.0 * torch.sin(v @ k.T + ph).sum(dim=1, keepdim=True)
    return (v * r).contiguous(), f.to(DEVICE).contiguous()


def _unit(d):
    return d / d.norm(dim=0, keepdim=True)


def _scattered(n, g, center, scale):
    """Rays from a sphere around the geometry toward uniform points of its box."""
    c = torch.tensor(center, device=DEVICE)[:, None]
    o = c + 2.0 * scale * _unit(torch.randn(3, n, device=DEVICE, generator=g))
    q = c + (_rand(g, 3, n) - 0.5) * scale
    return torch.cat([o, _unit(q - o)], 0).contiguous()


def _camera(n, g, eye, forward, tan):
    """Jittered pinhole rays in row order, about 16:9, looking along `forward` (an axis)."""
    w = max(1, int(round(math.sqrt(n * 16.0 / 9.0))))
    h = (n + w - 1) // w
    i = torch.arange(n, device=DEVICE)
    x = (((i % w).float() + _rand(g, n)) / w * 2 - 1) * tan * (w / h)
    y = (1 - ((i // w).float() + _rand(g, n)) / h * 2) * tan
    z = torch.full_like(x, forward)
    o = torch.tensor(eye, device=DEVICE)[:, None].expand(3, n)
    return torch.cat([o, _unit(torch.stack([x, y, z], 0))], 0).contiguous()


def _mesh_rays(case, g, rays):
    n = case["n_rays"]
    if case["geometry"] == "soup":
        mesh = F.InternalTriangleMesh(_soup(case["n_tri"], g))
        soa = _camera(n, g, (0.5, 0.5, -1.5), 1.0, 0.41421) if rays == "camera" else _scattered(n, g, (0.5,) * 3, 1.0)
    else:
        mesh = F.InternalTriangleMesh(*_sphere_mesh(case["level"], g))
        soa = _camera(n, g, (0.0, 0.0, 3.5), -1.0, 0.36397) if rays == "camera" else _scattered(n, g, (0.0,) * 3, 2.0)
    return mesh, soa


def _counts(case):
    """Log-uniform triangle counts of a batch, fixed by the case."""
    n = case["n_scenes"]
    lo, hi = math.log(case["low"]), math.log(case["high"])
    return [int(round(math.exp(lo + (hi - lo) * ((k * 0.6180339887498949) % 1.0)))) for k in range(n)]


def _noise(res, g):
    """Smooth density in [0, 4]: seeded random lattices, enlarged and summed."""
    rho = torch.zeros(1, 1, res, res, res, device=DEVICE)
    amp = 0.5
    for m in (5, 9, 17, 33):
        rho += amp * torch.nn.functional.interpolate(_rand(g, 1, 1, m, m, m), size=(res,) * 3, mode="trilinear",
                                                     align_corners=True)
        amp *= 0.5
    return (4.0 / 0.9375 * rho[0, 0]).contiguous()


def prepare(case, seed):
    g = _generator(seed)
    ctx = context()
    kind = case["kind"]
    st = {"case": case, "seed": seed}
    if kind in ("trace", "frame", "gradient"):
        mesh, soa = _mesh_rays(case, g, case.get("rays", "scatter"))
        b = F.RadixBVHBuilder(mesh, ctx)
        b.build()
        st.update(mesh=mesh, bvh=b, soa=soa, rays=F.Rays.from_soa(soa, tmin=1e-4))
        if kind == "gradient":
            n = case["n_rays"]
            st["dt"], st["du"], st["dv"] = (torch.randn(n, device=DEVICE, generator=g) for _ in range(3))
    elif kind == "shadow":
        # segments from surface points (hits of camera rays) to points of a light above
        mesh, soa = _mesh_rays(case, g, "camera")
        b = F.RadixBVHBuilder(mesh, ctx)
        b.build()
        h = b.intersect(F.Rays.from_soa(soa, tmin=1e-4))
        n = case["n_rays"]
        t = torch.where(h["prim"] >= 0, h["t"], _rand(g, n) * 2.0 + 1.0)
        p = soa[:3] + soa[3:] * t
        light = torch.stack([0.4 * _rand(g, n) - 0.2, torch.full((n,), 2.0, device=DEVICE), 0.4 * _rand(g, n) - 0.2], 0)
        d = light - p
        dist = d.norm(dim=0, keepdim=True)
        seg = torch.cat([p, d / dist, torch.full_like(dist, 1e-3), dist * 0.999], 0).contiguous()
        st.update(mesh=mesh, bvh=b, soa=seg, rays=F.Rays.from_soa(seg))
    elif kind == "batch":
        counts = _counts(case)
        offs, roffs = [0], [0]
        for c in counts:
            offs.append(offs[-1] + c)
            roffs.append(roffs[-1] + c * case["rays_per_tri"])
        mesh = F.InternalTriangleMesh(torch.cat([_soup(c, g) for c in counts], 0))
        soa = _scattered(roffs[-1], g, (0.5,) * 3, 1.0)
        b = F.BatchedRadixBVHBuilder(mesh, offs, ctx, node_width=4, leaf_size=case["leaf"])
        b.build()
        st.update(mesh=mesh, bvh=b, soa=soa, rays=F.Rays.from_soa(soa, tmin=1e-4), roffs=roffs)
    elif kind in ("volume", "scatter"):
        rho = _noise(case["res"], g)
        soa = _scattered(case["n_rays"], g, (0.5,) * 3, 1.0)
        if kind == "volume":
            vol = F.DenseGridVolume(rho, medium=F.Medium(0.8, 0.2, 0.3, 0.1, 0.0), ctx=ctx)
            st["dT"] = torch.randn(case["n_rays"], device=DEVICE, generator=g)
        else:
            rho = torch.where(rho > 2.2, rho - 2.2, torch.zeros_like(rho))  # clouds in empty space
            vol = F.SparseGridVolume.from_dense(rho, medium=F.Medium(8.0, 2.0, 0.3, 0.1, 0.0), ctx=ctx)
        st.update(vol=vol, soa=soa, rays=F.Rays.from_soa(soa))
    else:
        v, f = _sphere_mesh(case["level"], g)
        lv, lf = scenes.quad_light()
        pos = torch.cat([v, torch.from_numpy(lv).to(DEVICE)], 0).contiguous()
        ind = torch.cat([f, torch.from_numpy(lf).to(DEVICE) + v.shape[0]], 0).to(torch.int32).contiguous()
        b = F.RadixBVHBuilder(F.InternalTriangleMesh(pos, ind), ctx, node_width=4, leaf_size=2)
        b.build()
        st.update(bvh=b, light=f.shape[0], vol=None)
        if case["medium"]:
            st["vol"] = F.DenseGridVolume(0.2 * _noise(64, g), (-1.5,) * 3, (1.5,) * 3, F.Medium(0.8, 0.2, 0.3), ctx)
    return st


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "trace":
        return st["bvh"].intersect(st["rays"])
    if kind == "shadow":
        return st["bvh"].intersectP(st["rays"])
    if kind == "batch":
        if case["build_each"]:
            st["bvh"].build()
        return st["bvh"].intersect_batched(st["rays"], st["roffs"], persistent=2, refill_lanes=16, stack_depth=32)
    if kind == "frame":
        st["bvh"].build()
        return st["bvh"].intersect(st["rays"])
    if kind == "gradient":
        h = st["bvh"].intersect(st["rays"])
        return h, F.hit_adjoint(context(), st["mesh"], st["rays"], h, st["dt"], st["du"], st["dv"])
    if kind == "volume":
        T, ck = st["vol"].tr(st["rays"], st["seed"], checkpoint=True)
        return T, ck, st["vol"].tr_adjoint(st["rays"], st["seed"], st["dT"], T, ck)
    if kind == "scatter":
        return st["vol"].sample(st["rays"], st["seed"])
    img, rays = F.pathtrace(context(), st["bvh"], st["light"], 2, width=case["width"], height=case["height"],
                            spp=case["spp"], max_depth=case["max_depth"], volume=st["vol"], seed=st["seed"],
                            persistent=2, refill_lanes=16, **scenes.PATH_TRACING_CAMERA)
    return img, rays["closest_rays"], rays["shadow_rays"]


# ----------------------------------- work -----------------------------------

BYTES_PER_RAY = 24 + 16     # origin and direction in; prim, t, u, v out
BYTES_PER_TRI_BUILD = 268   # bounds 36, Morton 48, four sort passes 64, topology and refit 120


def _n_tri(case):
    if case["kind"] == "batch":
        return sum(_counts(case))
    return case["n_tri"] if case.get("geometry") == "soup" else 20 * 4 ** case["level"]


def work(case):
    """Bytes that have to move (rays in, results out, the triangles once, 268
    bytes per triangle of a build) and the arithmetic of one triangle test and
    of log4(n) four-wide box tests per ray, or of one tracking step per
    lattice cell that a ray crosses."""
    kind = case["kind"]
    if kind in ("volume", "scatter"):
        n, res = case["n_rays"], case["res"]
        grid = 4.0 * res ** 3
        steps = 4.0  # mean optical depth of a ray through the unit box, in majorant steps
        if kind == "volume":
            return {"bytes": n * (24 + 16) + grid + n * (24 + 20) + 2 * grid, "flops": n * steps * 2 * 60.0}
        return {"bytes": n * (24 + 17) + grid / 4, "flops": n * steps * 60.0}
    n_tri = _n_tri(case)
    tree = 48.0 * n_tri
    per_ray = 100.0 + 4 * 24.0 * math.log(max(n_tri, 4), 4)
    if kind == "render":
        n = case["width"] * case["height"] * case["spp"] * (1.0 + 0.5 * case["max_depth"])
        return {"bytes": n * BYTES_PER_RAY + tree, "flops": n * per_ray}
    n = n_tri * case["rays_per_tri"] if kind == "batch" else case["n_rays"]
    if kind == "shadow":
        return {"bytes": n * (32 + 1) + tree, "flops": n * per_ray}
    out = {"bytes": n * BYTES_PER_RAY + tree, "flops": n * per_ray}
    if kind == "frame" or case.get("build_each"):
        out["bytes"] += BYTES_PER_TRI_BUILD * n_tri
    if kind == "gradient":
        out["bytes"] += n * (24 + 12 + 12) + 36.0 * n_tri
        out["flops"] += n * 150.0
    return out


# ----------------------------------- exact -----------------------------------

MAX_PAIRS = 8e10


def _verts(mesh):
    p = mesh.p.double()
    i = mesh.ind.long() if mesh.ind is not None else torch.arange(p.shape[0], device=p.device).view(-1, 3)
    return p[i[:, 0]], p[i[:, 1]], p[i[:, 2]]


def _solve(o, d, a, b, c):
    """t, u, v of rays against triangles, row by row, in 64 bits."""
    e1, e2, s = b - a, c - a, o - a
    p = torch.linalg.cross(d, e2)
    det = (e1 * p).sum(-1)
    q = torch.linalg.cross(s, e1)
    return (e2 * q).sum(-1) / det, (s * p).sum(-1) / det, (d * q).sum(-1) / det


def _closest(mesh, soa, tmin):
    """Brute-force closest hit in 64 bits (prim, t, u, v): every quantity of a
    ray-triangle pair is linear in the triangle's coefficients, so the pairs
    of a block are matrix products."""
    a, b, c = _verts(mesh)
    o, d = soa[:3].double().T.contiguous(), soa[3:6].double().T.contiguous()
    n, m = o.shape[0], a.shape[0]
    nrm = torch.linalg.cross(b - a, c - a)
    mom = torch.linalg.cross(o, d)
    plu = torch.cat([d, mom], 1)                                   # Pluecker coordinates of the rays
    edge = [torch.cat([torch.linalg.cross(x, y), y - x], 1) for x, y in ((a, b), (b, c), (c, a))]
    nc = torch.cat([(a * nrm).sum(1, keepdim=True), -nrm], 1)
    o1 = torch.cat([torch.ones(n, 1, device=o.device, dtype=o.dtype), o], 1)
    best = torch.full((n,), math.inf, device=o.device, dtype=torch.float64)
    prim = torch.full((n,), -1, device=o.device, dtype=torch.int64)
    tb = 4096
    rb = max(1, min(n, (1 << 28) // min(m, tb)))
    for r0 in range(0, n, rb):
        r = slice(r0, min(n, r0 + rb))
        for t0 in range(0, m, tb):
            k = slice(t0, min(m, t0 + tb))
            s0 = plu[r] @ edge[0][k].T
            neg, pos = s0 <= 0, s0 >= 0
            for e in edge[1:]:
                s0 = plu[r] @ e[k].T
                neg &= s0 <= 0
                pos &= s0 >= 0
            neg |= pos
            t = (o1[r] @ nc[k].T) / (d[r] @ nrm[k].T)
            t = torch.where(neg & (t >= tmin), t, math.inf)
            lo, at = t.min(dim=1)
            near = lo < best[r]
            best[r] = torch.where(near, lo, best[r])
            prim[r] = torch.where(near, at + t0, prim[r])
    hit = prim >= 0
    k = prim.clamp(min=0)
    t, u, v = _solve(o, d, a[k], b[k], c[k])
    zero = torch.zeros_like(t)
    return prim, torch.where(hit, t, math.inf), torch.where(hit, u, zero), torch.where(hit, v, zero)


def exact(case, seed):
    if case["kind"] not in ("trace", "frame", "gradient") or float(_n_tri(case)) * case["n_rays"] > MAX_PAIRS:
        return None
    st = prepare(case, seed)
    prim, t, u, v = _closest(st["mesh"], st["soa"], 1e-4)
    hits = {"prim": prim, "t": t, "u": u, "v": v}
    if case["kind"] != "gradient":
        return hits
    # d(t, u, v)/d(vertices) of the fixed hits: M^T x = (dt, du, dv), M = [D, a - b, a - c]
    r = (prim >= 0).nonzero()[:, 0]
    a, b, c = (x[prim[r]] for x in _verts(st["mesh"]))
    d = st["soa"][3:6].double().T[r]
    c2, c3 = a - b, a - c
    x23, x31, x12 = torch.linalg.cross(c2, c3), torch.linalg.cross(c3, d), torch.linalg.cross(d, c2)
    det = (d * x23).sum(1, keepdim=True)
    gt, gu, gv = (st[k].double()[r][:, None] for k in ("dt", "du", "dv"))
    w = (x23 * gt + x31 * gu + x12 * gv) / det
    grad = torch.zeros(st["mesh"].p.shape, device=DEVICE, dtype=torch.float64)
    for j, wt in enumerate((1.0 - u[r] - v[r], u[r], v[r])):
        grad.index_add_(0, 3 * prim[r] + j, wt[:, None] * w)
    return hits, grad
