"""The tracking kernels at the edges of their work split and of the lattice:
ray counts around a warp and around a wave of resident warps, lattices from
two samples per axis to ones that end inside a brick, and gradient buffers
off the 16-byte grid."""
import numpy as np
import pytest
import torch

import geometry as G
import gpu_util as U

pytestmark = pytest.mark.gpu


class Medium:
    sigma_s, sigma_a, g, rr_threshold, majorant = 3.2, 0.8, 0.3, 0.1, 0.0


def _grid(shape):
    rng = np.random.default_rng(sum(shape))
    rho = rng.random(shape, dtype=np.float32) * 4.0
    if min(shape) > 8:
        rho[: 8, : 8, 8:] = 0.0  # an empty brick and part of its neighbours
    return rho


@pytest.mark.parametrize("n", [1, 31, 33, 4864 * 32 + 1])
@pytest.mark.parametrize("shape", [(2, 2, 2), (9, 8, 17), (33, 7, 5)])
def test_tracking_matches_oracle(ctx, oracle, shape, n):
    import fledge_gb300 as F
    rho = _grid(shape)
    r8 = G.sphere_rays(n, np.random.default_rng(n))
    rd, _ = U.rays_dev(r8)
    m = F.Medium(3.2, 0.8, 0.3)
    lo, hi = (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)
    To, cko = oracle.volume_tr(rho, lo, hi, Medium, r8, 5, want_ckpt=True)
    so = oracle.volume_sample(rho, lo, hi, Medium, r8, 6)
    for vol in (F.DenseGridVolume(U.dev(rho), lo, hi, m, ctx), F.SparseGridVolume.from_dense(U.dev(rho), lo, hi, m, ctx)):
        T, ck = vol.tr(rd, 5, checkpoint=True)
        assert np.array_equal(T.cpu().numpy(), To)
        assert np.array_equal(ck["k"].cpu().numpy().view(np.uint32), cko["k"])
        assert np.array_equal(ck["t"].cpu().numpy(), cko["t"]) and np.array_equal(ck["c"].cpu().numpy(), cko["c"])
        for a, b in zip(vol.sample(rd, 6), so):
            assert np.array_equal(a.cpu().numpy().reshape(-1), np.asarray(b).reshape(-1))
    ctx.sync()


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("shape", [(2, 2, 2), (9, 8, 17), (6, 7, 5)])
def test_adjoint_into_unaligned_buffers(ctx, oracle, shape, offset):
    """The gradient at every alignment, between guard values that stay."""
    import fledge_gb300 as F
    rho = _grid(shape)
    n = 3000
    r8 = G.sphere_rays(n, np.random.default_rng(9))
    rd, _ = U.rays_dev(r8)
    vol = F.DenseGridVolume(U.dev(rho), medium=F.Medium(3.2, 0.8, 0.3), ctx=ctx)
    T, ck = vol.tr(rd, 5, checkpoint=True)
    dL = U.dev(np.random.default_rng(10).standard_normal(n).astype(np.float32))
    buf = torch.full((rho.size + 8,), 7.0, device="cuda")
    grad = buf[offset:offset + rho.size].view(shape)
    grad.zero_()
    vol.tr_adjoint(rd, 5, dL, T, ck, grad)
    ctx.sync()
    ref = oracle.volume_tr_adjoint(rho, (0, 0, 0), (1, 1, 1), Medium, r8, 5, dL.cpu().numpy())
    g = grad.cpu().numpy().reshape(-1)
    scale = np.abs(ref).max()
    assert np.all(np.abs(g - np.asarray(ref).reshape(-1)) <= 1e-4 * scale)
    rest = torch.cat([buf[:offset], buf[offset + rho.size:]])
    assert bool((rest == 7.0).all())


@pytest.mark.parametrize("side_by_side", [True, False])
@pytest.mark.parametrize("over", [0, 1])
def test_many_rays(ctx, oracle, over, side_by_side):
    """On either side of the rule for warps of 256 rays: every ray's result is
    that of the same ray (the same stream) in the oracle, checked at the ends
    and in a seeded sample, and no ray is left out."""
    import fledge_gb300 as F
    n = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 8 * 512 + over
    rho = _grid((9, 8, 17))
    rng = np.random.default_rng(4)
    r8 = G.sphere_rays(n, rng)
    if side_by_side:
        r8[0:3] = np.array([[0.5], [0.5], [-2.0]], np.float32)
        d = np.stack([np.linspace(-0.3, 0.3, n), np.full(n, 0.05), np.ones(n)])
        r8[3:6] = d / np.linalg.norm(d, axis=0)
    r8 = r8.astype(np.float32)
    rd, _ = U.rays_dev(r8)
    vol = F.DenseGridVolume(U.dev(rho), medium=F.Medium(3.2, 0.8, 0.3), ctx=ctx)
    T, ck = vol.tr(rd, 5, checkpoint=True)
    T, k = T.cpu().numpy(), ck["k"].cpu().numpy().view(np.uint32)
    ok = vol.sample(rd, 6)[0].cpu().numpy()
    To, cko = oracle.volume_tr(rho, (0.0,) * 3, (1.0,) * 3, Medium, r8, 5, want_ckpt=True)
    so = np.asarray(oracle.volume_sample(rho, (0.0,) * 3, (1.0,) * 3, Medium, r8, 6)[0])
    assert np.array_equal(T, To) and np.array_equal(k, cko["k"]) and np.array_equal(ok.reshape(-1), so.reshape(-1))
    ctx.sync()
