"""The 4-wide quantised layout where its boxes, its stack or its tie rules
could go wrong: the hits must still be those of the exact boxes (oracle DEV
arithmetic: ids equal but for exact ties, t/u/v bit-equal where they agree;
occlusion bits equal)."""
import numpy as np
import pytest

import geometry as G
import gpu_util as U

pytestmark = pytest.mark.gpu


def _scene(kind):
    rng = np.random.default_rng(404)
    pos = G.random_soup(3000, rng, half=0.05).reshape(-1, 3, 3)
    rays = G.sphere_rays(20000, rng)
    if kind == "duplicates":          # every hit is an exact tie, within and across leaf ranges
        pos = np.concatenate([pos, pos, pos[::-1]])
    elif kind == "planes":            # overlapping axis-aligned triangles: flat boxes, equal and nearly equal t
        pos[:, :, 2] = np.float32(0.25) * np.round(4 * pos[:, :1, 2])
    elif kind == "far":               # coordinates large against the boxes
        pos += np.float32(4096.0)
        rays[0:3] += np.float32(4096.0)
    elif kind == "axis":              # zero direction components
        a = rng.integers(0, 3, rays.shape[1])
        rays[3:6] = 0.0
        rays[3 + a, np.arange(rays.shape[1])] = np.where(rng.random(rays.shape[1]) < 0.5, 1.0, -1.0)
        rays[0:3] = rng.random((3, rays.shape[1])) * 1.2 - 0.1
    elif kind == "tiny":
        pos *= np.float32(2.0 ** -24)
        rays[0:3] *= np.float32(2.0 ** -24)
        rays[6] = 0.0
    elif kind == "huge":              # the distances' numerators still fit fp32
        pos *= np.float32(2.0 ** 30)
        rays[0:3] *= np.float32(2.0 ** 30)
    elif kind == "nonfinite":         # a box without bounds above every other one
        pos[7, 1] = (np.inf, 0.5, -np.inf)
        pos[8] = np.nan
    elif kind == "slivers":           # the stack leaves shared memory
        pos, rays = G.sliver_comb(64, rng)
    return np.ascontiguousarray(pos.reshape(-1, 3).astype(np.float32)), rays.astype(np.float32)


KINDS = ["duplicates", "planes", "far", "axis", "tiny", "huge", "nonfinite", "slivers"]


@pytest.mark.parametrize("leaf", [1, 3, 8])
@pytest.mark.parametrize("kind", KINDS)
def test_quantised_boxes_change_no_hit(ctx, oracle, kind, leaf):
    pos, r8 = _scene(kind)
    b, _ = U.gpu_build(ctx, pos, width=4, leaf=leaf)
    exact, _ = U.gpu_build(ctx, pos, width=8, leaf=leaf)  # fp32 boxes
    rd, _ = U.rays_dev(r8)
    hg, he = U.host(b.intersect(rd)), U.host(exact.intersect(rd))
    occ, occ_e = b.intersectP(rd).cpu().numpy(), exact.intersectP(rd).cpu().numpy()
    ctx.sync()
    if kind == "nonfinite":  # the oracle's Morton codes of such a scene are its own
        tri = pos.reshape(-1, 3, 3)
        diff = np.nonzero(hg["prim"] != he["prim"])[0]
        for i in diff:
            k = [oracle.pluecker(tri[p, 0], tri[p, 1], tri[p, 2], r8[0:3, i], r8[3:6, i], oracle.MODE_DEV)
                 for p in (hg["prim"][i], he["prim"][i]) if p >= 0]
            assert len(k) == 2 and k[0][0] and k[1][0] and k[0][1][0] == k[1][1][0], i
        assert np.array_equal(occ, occ_e)
        return
    tree = oracle.build_bvh(pos)
    bad, ties, ho = U.compare_closest(oracle, pos, None, tree, r8, hg, oracle.MODE_DEV)
    extra = 0
    if leaf > 1:  # hits that a leaf range's box lets in and the reference's tighter boxes keep out
        extra = np.count_nonzero((hg["prim"] >= 0) & (ho["prim"] < 0))
        assert extra == np.count_nonzero((he["prim"] >= 0) & (ho["prim"] < 0))
    if kind != "planes":  # there the order of visits decides between nearly equal t
        assert bad == extra, (bad, ties, extra)
    same = hg["prim"] == ho["prim"]
    for k in ("t", "u", "v"):
        assert np.array_equal(hg[k][same], ho[k][same]), k
    assert np.array_equal(hg["prim"] >= 0, he["prim"] >= 0) and np.array_equal(occ, occ_e)


def _directions(kind, v, n, rng):
    """Unit rays through the unit cube whose direction has a zero or a very
    small component, or a very small or large length."""
    r = np.zeros((8, n), np.float32)
    if kind == "sphere":
        r[:] = G.sphere_rays(n, rng)
    else:  # down the z axis from above, or from inside
        r[0:3] = rng.random((3, n))
        r[2, ::2] = 2.0
        r[5] = -1.0
    if kind == "tilt":
        r[3] = v
    else:
        r[3:6] *= np.float32(v)
    r[6], r[7] = 0.0, np.inf
    return r


@pytest.mark.parametrize("scale", [1.0, 1e3, 1e6, 1.1e9, 4e9, 1e12, 1e18])
@pytest.mark.parametrize("kind,v", [("axis", 1.0), ("axis", 1e-14), ("axis", 1e-28), ("axis", 1e31), ("sphere", 1e-36),
                                    ("sphere", 1e31), ("tilt", 1e-10), ("tilt", 6e-17), ("tilt", 1e-33),
                                    ("tilt", 5e-37), ("tilt", 1e-38), ("tilt", 1e-40)])
def test_inverse_directions_at_the_ends_of_fp32(ctx, oracle, scale, kind, v):
    """Distances to quantised planes that would overflow or lose their bits:
    the hits stay those of fp32 boxes, for closest and any hit.  One scene is as
    thick as it is wide, the other a millionth of that along x."""
    rng = np.random.default_rng(91)
    for thin in (False, True):
        pos = G.random_soup(3000, rng, half=0.05).reshape(-1, 3)
        r8 = _directions(kind, v, 20000, rng)
        if thin:
            pos[:, 0] = (pos[:, 0] - np.float32(0.5)) * np.float32(1e-6)
            r8[0] = (r8[0] - np.float32(0.5)) * np.float32(1e-6)
        pos *= np.float32(scale)
        r8[0:3] *= np.float32(scale)
        b, _ = U.gpu_build(ctx, pos, width=4)
        exact, _ = U.gpu_build(ctx, pos, width=8)
        rd, _ = U.rays_dev(r8)
        hg, he = U.host(b.intersect(rd)), U.host(exact.intersect(rd))
        occ, occ_e = b.intersectP(rd).cpu().numpy(), exact.intersectP(rd).cpu().numpy()
        ctx.sync()
        assert np.array_equal(hg["prim"] >= 0, he["prim"] >= 0), (thin, np.count_nonzero(hg["prim"] >= 0))
        assert np.array_equal(occ, occ_e), thin
        tri = pos.reshape(-1, 3, 3)
        for i in np.nonzero(hg["prim"] != he["prim"])[0]:  # at the same distance, else not another triangle
            t = [oracle.pluecker(*tri[p], r8[0:3, i], r8[3:6, i], oracle.MODE_DEV)[1][0]
                 for p in (hg["prim"][i], he["prim"][i])]
            assert t[0] == t[1], (thin, i)
        same = hg["prim"] == he["prim"]
        for k in ("t", "u", "v"):
            assert np.array_equal(hg[k][same], he[k][same], equal_nan=True), (thin, k)
    if kind != "sphere" and abs(np.log10(v)) < 15 and scale < 1e12:
        assert (hg["prim"] >= 0).mean() > 0.1


def test_hits_in_front_of_their_own_box(ctx, oracle):
    """Two triangles per scene: a sliver of 1e-7 to 1e-6 along the ray, whose
    fp32 t may lie well in front of its box, and a triangle across the ray about
    where that box begins.  Which box the ray enters first, and whether the
    other one begins beyond that hit, decides, as with fp32 boxes (8-wide;
    distances that agree but for the bits which the child's number replaces may
    be in either order)."""
    import fledge_gb300 as F
    n = 1 << 17
    rng = np.random.default_rng(5)
    d = np.zeros((n, 3))
    d[np.arange(n), rng.integers(0, 3, n)] = 1.0
    d += 0.3 * (rng.random((n, 3)) - 0.5)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = rng.random((n, 3))
    u = np.cross(d, [0.37, 0.61, 0.7])
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = np.cross(d, u)
    s = 1e-7 * 10.0 ** rng.random((n, 1))
    ang = 2 * np.pi * rng.random((n, 1))

    def corner(k, t, r):
        x = ang + 2 * np.pi / 3 * k
        return o + t * d + r * (np.cos(x) * u + np.sin(x) * v)

    along = 0.2 * (rng.random((n, 3)) - 0.5)
    across = 1 + along.min(1, keepdims=True) + (rng.random((n, 1)) - 0.8) * np.exp(9 * rng.random((n, 1)) - 13)
    tri = np.stack([np.stack([corner(k, 1 + along[:, k:k + 1], s) for k in range(3)], 1),
                    np.stack([corner(k, across, 0.01) for k in range(3)], 1)], 1).astype(np.float32)
    r8 = np.zeros((8, n), np.float32)
    r8[0:3], r8[3:6], r8[7] = o.T, d.T, np.inf
    rd, _ = U.rays_dev(r8)
    hits = []
    for w in (4, 8):
        b = F.BatchedRadixBVHBuilder(F.InternalTriangleMesh(U.dev(tri.reshape(-1, 3))), 2 * np.arange(n + 1), ctx, node_width=w)
        b.build()
        hits.append(U.host(b.intersect_batched(rd, np.arange(n + 1))))
    ctx.sync()
    assert (hits[1]["prim"] == 0).sum() > 100
    inv = np.float32(1) / r8[3:6].T
    planes = (np.where(inv[:, None] < 0, tri.max(2), tri.min(2)) - r8[0:3].T[:, None]) * inv[:, None]
    near = np.maximum(planes.max(2), np.float32(0)).view(np.int32)
    same = hits[0]["prim"] == hits[1]["prim"]
    assert np.count_nonzero(~same) < 100
    for i in np.nonzero(~same)[0]:
        t = [np.float32(oracle.pluecker(*tri[i, k], r8[0:3, i], r8[3:6, i], oracle.MODE_DEV)[1][0]).view(np.int32)
             for k in (0, 1)]
        assert min(abs(near[i, 0] - near[i, 1]), abs(near[i, 0] - t[1]), abs(near[i, 1] - t[0])) < 8, i
    for k in ("t", "u", "v"):
        assert np.array_equal(hits[0][k][same], hits[1][k][same]), k


@pytest.mark.parametrize("leaf", [1, 3, 8])
@pytest.mark.parametrize("kind", ["soup", "copies3", "copies7", "copies9", "duplicates", "planes", "quads", "slivers"])
def test_ids_are_those_of_the_walk_over_exact_boxes(ctx, kind, leaf):
    """Directions 2^104 times as long take every ray over the exact boxes, with
    all its arithmetic scaled by a power of two: the same ids (and distances, but
    for the last bit: the low parts of their refinement become subnormal), also
    where several triangles share the closest distance and the order of visits
    decides (`copies<k>`: k equal triangles each, next to each other or not)."""
    import fledge_gb300 as F
    import torch
    rng = np.random.default_rng(58)
    rays = G.sphere_rays(200000, rng)
    if kind.startswith("copies"):
        tri = G.random_soup(1500, rng, half=0.05).reshape(-1, 9)
        k = int(kind[6:])
        pos = np.concatenate([np.repeat(tri[:750], k, 0), np.tile(tri[750:], (k, 1))])
    elif kind == "quads":  # layers of squares, their diagonals and edges shared
        x, y, z = np.meshgrid(np.arange(24) / 24, np.arange(24) / 24, (0.1, 0.3, 0.5, 0.7), indexing="ij")
        c = [np.stack([x.ravel() + i / 24, y.ravel() + j / 24, z.ravel()], 1) for i, j in ((0, 0), (1, 0), (1, 1), (0, 1))]
        pos = np.concatenate([np.concatenate([c[0], c[1], c[2]], 1), np.concatenate([c[0], c[2], c[3]], 1)])
        rays[0:2, ::2] = rng.integers(0, 49, (2, 100000)) / 48  # every other one straight down through corners and edges
        rays[2, ::2], rays[3:5, ::2], rays[5, ::2] = 2.0, 0.0, -1.0
    elif kind == "slivers":
        pos, rays = G.sliver_comb(64, rng)
    else:
        pos = G.random_soup(3000, rng, half=0.05) if kind == "soup" else _scene(kind)[0]
    b, _ = U.gpu_build(ctx, np.ascontiguousarray(pos.reshape(-1, 3), np.float32), width=4, leaf=leaf)
    rays = rays.astype(np.float32)
    rays[6] = 0.0
    long = rays.copy()
    long[3:6] *= np.float32(2.0 ** 104)
    (rd, _), (rl, _) = U.rays_dev(rays), U.rays_dev(long)
    h, e = b.intersect(rd), b.intersect(rl)
    ctx.sync()
    assert (h["prim"] >= 0).float().mean() > 0.1
    assert torch.equal(h["prim"], e["prim"]), int((h["prim"] != e["prim"]).sum())
    hit = h["prim"] >= 0
    assert ((h["t"] - e["t"] * 2.0 ** 104).abs() <= 2.0 ** -23 * h["t"])[hit].all()
    assert torch.equal(b.intersectP(rd), b.intersectP(rl))


@pytest.mark.parametrize("leaf", [1, 2, 3, 8])
@pytest.mark.parametrize("distance", [3.0, 30.0, 300.0])
def test_rays_at_the_vertices_of_a_mesh(ctx, distance, leaf):
    """Rays at the vertices of a displaced sphere of 81,920 triangles, half of them
    off by up to 1e-6: the triangles around a vertex share its distance but for
    rounding, which also puts some of the distances before their boxes.  The
    same ids as by the walk over exact boxes (directions 2^104 times as long)."""
    import fledge_gb300 as F
    import torch
    from fledge_gb300 import scenes
    v, f = scenes.icosphere(6, amplitude=0.05)
    g = torch.Generator(device="cuda").manual_seed(int(distance))
    n = 1 << 20
    p, ind = U.dev(v.astype(np.float32)), U.dev(f.astype(np.int32))
    o = torch.randn(3, n, device="cuda", generator=g)
    o = o / o.norm(dim=0) * distance
    at = p[torch.randint(0, p.shape[0], (n,), device="cuda", generator=g)].T
    at = at + (torch.rand(3, n, device="cuda", generator=g) - 0.5) * 2e-6 * (torch.arange(n, device="cuda") % 2)
    d = at - o
    d = d / d.norm(dim=0)
    b = F.RadixBVHBuilder(F.InternalTriangleMesh(p, ind), ctx, leaf_size=leaf)
    b.build()
    r, rl = (F.Rays.from_soa(torch.cat([o, d * k], 0).contiguous(), tmin=0.0) for k in (1.0, 2.0 ** 104))
    h, e = b.intersect(r)["prim"], b.intersect(rl)["prim"]
    ctx.sync()
    assert (h >= 0).float().mean() > 0.9
    assert torch.equal(h, e), int((h != e).sum())
    assert torch.equal(b.intersectP(r), b.intersectP(rl))


@pytest.mark.parametrize("leaf", [1, 2, 3, 8])
@pytest.mark.parametrize("kind", ["flat", "inside"])
def test_rays_nearly_along_an_axis_at_the_vertices(ctx, kind, leaf):
    """Rays at the vertices of a height field whose direction has a component of
    about 1e-3 along x (`flat`): a triangle hit by rounding beside its box may be
    one that the ray leaves along that axis well before the hit.  The same ids as by the walk over exact boxes (directions 2^104 times
    as long)."""
    import fledge_gb300 as F
    import torch
    m, n = 256, 1 << 21
    g = torch.Generator(device="cuda").manual_seed(17)
    x, y = torch.meshgrid(torch.arange(m + 1, device="cuda") / m, torch.arange(m + 1, device="cuda") / m, indexing="ij")
    p = torch.stack([x, y, 0.1 * torch.sin(11 * x) * torch.cos(7 * y)], -1).reshape(-1, 3).contiguous()
    i = (torch.arange(m, device="cuda")[:, None] * (m + 1) + torch.arange(m, device="cuda")).reshape(-1)
    f = torch.cat([torch.stack([i, i + m + 1, i + m + 2], 1), torch.stack([i, i + m + 2, i + 1], 1)]).int().contiguous()
    d = torch.randn(n, 3, device="cuda", generator=g)
    if kind == "flat":
        d[:, 0] *= 1e-3
    d = d / d.norm(dim=1, keepdim=True)
    back = 0.3 * torch.rand(n, 1, device="cuda", generator=g) if kind == "inside" else 3.0
    o = p[torch.randint(0, p.shape[0], (n,), device="cuda", generator=g)] - back * d
    b = F.RadixBVHBuilder(F.InternalTriangleMesh(p, f), ctx, leaf_size=leaf)
    b.build()
    r, rl = (F.Rays.from_soa(torch.cat([o.T, d.T * k], 0).contiguous(), tmin=0.0) for k in (1.0, 2.0 ** 104))
    h, e = b.intersect(r)["prim"], b.intersect(rl)["prim"]
    ctx.sync()
    assert (h >= 0).float().mean() > 0.9
    assert torch.equal(h, e), int((h != e).sum())
    assert torch.equal(b.intersectP(r), b.intersectP(rl))


def test_more_ties_than_the_list_holds(ctx):
    """Over 2^20 rays that all end in a tie: the list overflows and the rays
    are found by their marks.  Equal to tracing them in parts."""
    import fledge_gb300 as F
    import torch
    pos, _ = _scene("duplicates")
    b, _ = U.gpu_build(ctx, pos, width=4, leaf=1)
    soa = F.gen_rays(ctx, 3 << 19, 77)
    soa[3:6] = 0.5 - soa[0:3] + 0.2 * (soa[3:6] - 0.5)  # toward the middle: nearly all hit
    whole = b.intersect(F.Rays.from_soa(soa))
    assert int((whole["prim"] >= 0).sum()) > 1 << 20
    for a in range(0, soa.shape[1], 1 << 19):
        part = b.intersect(F.Rays.from_soa(soa[:, a:a + (1 << 19)].contiguous()))
        for k in part:
            assert torch.equal(part[k], whole[k][a:a + (1 << 19)]), k
    ctx.sync()


@pytest.mark.parametrize("n", [1, 31, 33, 4863, 4865, 155649])
def test_small_batches_spread_over_warps(ctx, oracle, n):
    """Ray counts around the edges of the spread of a small batch over warps
    and blocks: equal to the same rays inside a large batch."""
    import fledge_gb300 as F
    import torch
    pos = F.gen_triangles(ctx, 5000, 12)
    b = F.RadixBVHBuilder(F.InternalTriangleMesh(pos), ctx)
    b.build()
    soa = F.gen_rays(ctx, 300000, 13)
    whole = b.intersect(F.Rays.from_soa(soa))
    occ = b.intersectP(F.Rays.from_soa(soa))
    part = F.Rays.from_soa(soa[:, :n].contiguous())
    hp = b.intersect(part)
    for k in hp:
        assert torch.equal(hp[k], whole[k][:n]), k
    assert torch.equal(b.intersectP(part), occ[:n])
    ctx.sync()


def test_one_triangle_scenes_of_a_batch(ctx, oracle):
    """Scenes of no, one and two triangles in one 4-wide batch, also after a
    change of width: each equal to its own handle."""
    import fledge_gb300 as F
    import torch
    counts = [1, 0, 2, 1, 1, 600, 1]
    offs = np.concatenate([[0], np.cumsum(counts)])
    pos = F.gen_triangles(ctx, int(offs[-1]), 5, half_extent=0.3)
    per = 2000
    soa = F.gen_rays(ctx, per * len(counts), 6)
    bb = F.BatchedRadixBVHBuilder(F.InternalTriangleMesh(pos), offs, ctx, node_width=8)
    bb.build()
    bb.set_width(4)
    h = bb.intersect_batched(F.Rays.from_soa(soa), per * np.arange(len(counts) + 1))
    for s, c in enumerate(counts):
        one = F.RadixBVHBuilder(F.InternalTriangleMesh(pos[3 * offs[s]:3 * offs[s + 1]].contiguous()), ctx, node_width=2)
        one.build()
        r = F.Rays.from_soa(soa[:, per * s:per * (s + 1)].contiguous())
        ho = one.intersect(r)
        for k in ho:
            assert torch.equal(ho[k], h[k][per * s:per * (s + 1)]), (s, k)
        four = F.RadixBVHBuilder(one.mesh, ctx, node_width=4)
        four.build()
        assert torch.equal(four.intersectP(r), one.intersectP(r))
    ctx.sync()


@pytest.mark.parametrize("over", [0, 1])
def test_where_settling_also_finishes(ctx, oracle, over):
    """On either side of the rule that lets one kernel settle and finish:
    every hit a tie, closest and any hit in turn on the counters that the trace
    before them has cleared."""
    import torch
    pos, _ = _scene("duplicates")
    n = torch.cuda.get_device_properties(0).multi_processor_count * 384 + over
    r8 = G.sphere_rays(n, np.random.default_rng(12))
    b, _ = U.gpu_build(ctx, pos, width=4)
    rd, _ = U.rays_dev(r8)
    tree = oracle.build_bvh(pos)
    for _ in range(3):
        h = U.host(b.intersect(rd))
        occ = b.intersectP(rd).cpu().numpy()
        bad, _, ho = U.compare_closest(oracle, pos, None, tree, r8, h, oracle.MODE_DEV)
        assert bad == 0
        same = h["prim"] == ho["prim"]
        assert np.array_equal(h["t"][same], ho["t"][same])
        assert np.array_equal(occ != 0, ho["prim"] >= 0)
    ctx.sync()


@pytest.mark.parametrize("over", [0, 1])
def test_where_settling_changes_its_blocks(ctx, over):
    """On either side of the 2^21 rays above which the settling kernel runs in
    other blocks, among them more ties than its list holds and few: equal to
    tracing the rays in parts."""
    import fledge_gb300 as F
    import torch
    n = (1 << 21) + over
    soa = F.gen_rays(ctx, n, 78)
    soa[3:6] = 0.5 - soa[0:3] + 0.2 * (soa[3:6] - 0.5)
    for kind in ("duplicates", "planes"):
        b, _ = U.gpu_build(ctx, _scene(kind)[0], width=4, leaf=1)
        whole = b.intersect(F.Rays.from_soa(soa))
        occ = b.intersectP(F.Rays.from_soa(soa))
        for a in range(0, n, 700001):
            r = F.Rays.from_soa(soa[:, a:a + 700001].contiguous())
            part = b.intersect(r)
            for k in part:
                assert torch.equal(part[k], whole[k][a:a + 700001]), (kind, k)
            assert torch.equal(b.intersectP(r), occ[a:a + 700001]), kind
        ctx.sync()


def test_a_walk_of_more_than_2_to_22_entries(ctx):
    """A ray over the exact boxes (its direction is too long for the quantised
    ones) that enters the boxes of 3.4 million equal triangles before the one
    that it hits: the walk, about 4 s long, is not cut short."""
    import fledge_gb300 as F
    import torch
    n = 3400000
    pos = torch.tensor([[0.0, 0, 0.1], [1, 0, 3], [0, 1, 3]], device="cuda").repeat(n + 1, 1)
    pos[3 * n:] = torch.tensor([[0.2, 0.2, 1.0], [0.6, 0.2, 1], [0.2, 0.6, 1]], device="cuda")
    b = F.RadixBVHBuilder(F.InternalTriangleMesh(pos), ctx)
    b.build()
    r = torch.tensor([[0.3], [0.3], [-1.0], [0.0], [0.0], [2.0 ** 103]], device="cuda")
    h = b.intersect(F.Rays.from_soa(r, tmin=0.0))
    ctx.sync()
    assert int(h["prim"][0]) == n and float(h["t"][0]) == 2.0 ** -102


@pytest.mark.parametrize("scenes", [1, 5])
def test_the_tuner_tries_nothing_twice(ctx, scenes):
    """Every trial on the 4-wide layout differs from the others in something
    that its kernel reads: leaf ranges, refills up to 8 lanes, the block size, the
    ray sort."""
    import ctypes as C
    import json

    import fledge_gb300 as F
    offs = np.arange(scenes + 1, dtype=np.int64) * 4000
    mesh = F.InternalTriangleMesh(F.gen_triangles(ctx, int(offs[-1]), 21))
    rays = F.Rays.from_soa(F.gen_rays(ctx, 10 * int(offs[-1]), 22), tmin=1e-4)
    best, w, leaf, buf, r = F.FlgTraceOpts(), C.c_int32(), C.c_int32(), C.create_string_buffer(1 << 16), rays.struct()
    if scenes == 1:
        b = F.RadixBVHBuilder(mesh, ctx)
        b.build()
        ctx.check(ctx.lib.flg_autotune_trace(ctx.h, b.h, C.byref(r), rays.n, C.byref(best), C.byref(w), buf, len(buf)))
    else:
        b = F.BatchedRadixBVHBuilder(mesh, offs, ctx)
        b.build()
        ro = np.ascontiguousarray(10 * offs)
        ctx.check(ctx.lib.flg_autotune_trace_batched(ctx.h, b.h, C.byref(r), ro.ctypes.data_as(C.POINTER(C.c_int64)), 3,
                                                     C.byref(best), C.byref(w), C.byref(leaf), buf, len(buf)))
    four = [(t["leaf_size"], min(t["refill_lanes"], 8), t["block_threads"], t["ray_sort"])
            for t in json.loads(buf.value.decode())["trials"] if t["node_width"] == 4]
    assert w.value == 4 and len(four) > 6
    assert len(set(four)) == len(four), four
