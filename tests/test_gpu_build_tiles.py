"""Builds at the edges of the sort tiles (1024 pairs, or 3072 once those give
every SM a tile), of the scene-bounds chunks and of the collapse's claims:
one scene, batches below and above the rule for sorting scenes in their own
runs of tiles, and captured builds of both layouts."""
import ctypes as C

import numpy as np
import pytest
import torch

import geometry as G
import gpu_util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [127, 129, 1023, 1024, 1025, 3072, 4097])
def test_build_at_tile_edges(ctx, oracle, n):
    pos = G.random_soup(n, np.random.default_rng(n))
    b, _ = U.gpu_build(ctx, pos)
    for _ in range(2):  # a rebuild starts from what the first left behind
        U.assert_same_topology(b.topology(), oracle.build_bvh(pos))
        b.build()


@pytest.mark.parametrize("more", [-1, 0, 1])
def test_build_where_the_tile_changes(ctx, oracle, more):
    n = torch.cuda.get_device_properties(0).multi_processor_count * 3072 + more
    pos = G.random_soup(n, np.random.default_rng(7), half=0.003)
    b, _ = U.gpu_build(ctx, pos)
    U.assert_same_topology(b.topology(), oracle.build_bvh(pos))


@pytest.mark.parametrize("counts", [
    [1024, 1025, 0, 1, 1023, 2048, 2],       # below 4 tiles of 1024 per scene: one sort with a scene pass
    [16384, 0, 1, 1024, 1025, 20000, 2, 0],  # above: each scene in its own tiles
    [4096, 4096], [4096, 4095],              # on either side of the rule
])
def test_batched_build_at_tile_edges(ctx, oracle, counts):
    import fledge_gb300 as F
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    pos = G.random_soup(int(offs[-1]), np.random.default_rng(31))
    bb = F.BatchedRadixBVHBuilder(F.InternalTriangleMesh(U.dev(pos)), offs, ctx, node_width=2)
    for _ in range(2):
        bb.build()
        for s, c in enumerate(counts):
            if c:
                U.assert_same_topology(bb.topology(s), oracle.build_bvh(pos[3 * offs[s]:3 * offs[s + 1]]))


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("counts", [[2], [5], [129], [20001], [300, 1, 0, 2, 5000, 33]])
def test_captured_build_traces_like_the_oracle(oracle, width, counts):
    """One cooperative collapse, also inside a captured graph."""
    import fledge_gb300 as F
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    rng = np.random.default_rng(11)
    first = U.dev(G.random_soup(int(offs[-1]), rng, half=0.1))
    pos = first.clone()
    per = 1000
    roff = np.arange(len(counts) + 1, dtype=np.int64) * per
    r8 = G.sphere_rays(per * len(counts), rng)
    rays, _ = U.rays_dev(r8)
    s = torch.cuda.Stream()
    ctx2 = F.Context(0, s)
    b = F.BatchedRadixBVHBuilder(F.InternalTriangleMesh(pos), offs, ctx2, node_width=width)
    with torch.cuda.stream(s):
        b.build()
        b.intersect_batched(rays, roff)
        g = C.c_void_p()
        ctx2.check(ctx2.lib.flg_graph_begin(ctx2.h))
        ctx2.check(ctx2.lib.flg_bvh_rebuild(ctx2.h, b.h, C.c_void_p(pos.data_ptr())))
        ctx2.check(ctx2.lib.flg_graph_end(ctx2.h, C.byref(g)))
    ctx2.sync()
    for trial in range(3):
        new = G.random_soup(int(offs[-1]), np.random.default_rng(100 + trial), half=0.1)
        pos.copy_(U.dev(new))
        torch.cuda.synchronize()
        ctx2.check(ctx2.lib.flg_graph_launch(ctx2.h, g))
        with torch.cuda.stream(s):
            h = U.host(b.intersect_batched(rays, roff))
        for k, c in enumerate(counts):
            part = {q: v[k * per:(k + 1) * per] for q, v in h.items()}
            if c < 2:
                continue
            tri = new[3 * offs[k]:3 * offs[k + 1]]
            bad, _, _ = U.compare_closest(oracle, tri, None, oracle.build_bvh(tri), r8[:, k * per:(k + 1) * per], part,
                                          oracle.MODE_DEV)
            assert bad == 0, (trial, k)
    ctx2.lib.flg_graph_destroy(g)
    ctx2.close()


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("n", [(1 << 20), (1 << 20) + 1])
def test_either_collapse_of_a_scene(ctx, width, n):
    """On either side of the rule for collapsing in subtrees: the hits of the
    binary tree, which has none to collapse."""
    import fledge_gb300 as F
    pos = F.gen_triangles(ctx, n, 21)
    rays = F.Rays.from_soa(F.gen_rays(ctx, 20000, 22), tmin=1e-4)
    out = []
    for w in (2, width):
        b = F.RadixBVHBuilder(F.InternalTriangleMesh(pos), ctx, node_width=w)
        b.build()
        b.build()
        out.append(U.host(b.intersect(rays)))
    ctx.sync()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("scenes", [1024, 1025])
def test_either_collapse_of_a_batch(ctx, scenes):
    import fledge_gb300 as F
    rng = np.random.default_rng(5)
    counts = rng.integers(0, 40, scenes)
    counts[7] = 3000
    counts[counts < 2] = 2  # as many roots as scenes
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    roff = np.arange(scenes + 1, dtype=np.int64) * 20
    pos = U.dev(G.random_soup(int(offs[-1]), rng, half=0.1))
    rays, _ = U.rays_dev(G.sphere_rays(int(roff[-1]), rng))
    out = []
    for w in (2, 4):
        b = F.BatchedRadixBVHBuilder(F.InternalTriangleMesh(pos), offs, ctx, node_width=w)
        b.build()
        b.build()
        out.append(U.host(b.intersect_batched(rays, roff)))
    ctx.sync()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("n", [1, 2, 2048, 2049, 8193, 16384, 16385, 20001, 32767, 32768, 32769])
def test_cluster_sort_edges(ctx, oracle, n):
    """Cluster sizes, positions per thread and the last size of the sort in one
    cluster; the second scene has only three different codes."""
    for pos in (G.random_soup(n, np.random.default_rng(n)),
                np.tile(G.random_soup(3, np.random.default_rng(1)), ((n + 2) // 3, 1))[:3 * n]):
        b, _ = U.gpu_build(ctx, pos)
        b.build()
        if n > 1:
            U.assert_same_topology(b.topology(), oracle.build_bvh(pos))
    ctx.sync()


@pytest.mark.parametrize("counts", [[40000], [33000, 40000, 500]])
def test_scene_bounds_with_negative_zeros(ctx, oracle, counts):
    """-0 as the extreme of most blocks' triangles, beside a negative minimum and
    as the largest coordinate of an axis: the bounds, and so the codes, are the
    oracle's."""
    import fledge_gb300 as F
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    tri = np.random.default_rng(5).random((int(offs[-1]), 3, 3)).astype(np.float32)
    tri[::7, 0, 0] = np.float32(-0.0)
    tri[:, :, 1] = -tri[:, :, 1]
    tri[::5, 1, 1] = np.float32(-0.0)
    tri[offs[:-1] + 3, 1, 0] = np.float32(-0.25)
    pos = tri.reshape(-1, 3)
    if len(counts) == 1:
        b, _ = U.gpu_build(ctx, pos)
    else:
        b = F.BatchedRadixBVHBuilder(F.InternalTriangleMesh(U.dev(pos)), offs, ctx, node_width=2)
    for _ in range(3):
        b.build()
        for s in range(len(counts)):
            U.assert_same_topology(b.topology(s), oracle.build_bvh(pos[3 * offs[s]:3 * offs[s + 1]]))
