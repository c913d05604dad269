"""Halton digits of large sample indices: direct lighting alone, where no path
can part from the oracle's by an ulp of a bounce direction.  (The number of
bounces can: whether one at the rim of the sampled disk has pdf 0 takes the
last bit of cos and sin.)"""
import numpy as np
import pytest

from fledge_gb300.scenes import icosphere, quad_light

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,spp", [(16, 12, 300), (3, 130, 40), (130, 1, 40), (1, 1, 1000)])
def test_many_samples_match_oracle(ctx, oracle, W, H, spp):
    import fledge_gb300 as F
    import gpu_util as U
    v, f = icosphere(3)
    lv, lf = quad_light()
    pos, ind = np.concatenate([v, lv], 0), np.concatenate([f, lf + len(v)], 0)
    b, _ = U.gpu_build(ctx, pos, ind, width=4)
    cam = dict(eye=(0.0, 0.6, 3.5), target=(0.0, 0.0, 0.0), up=(0.0, 1.0, 0.0), fov_deg=40.0)
    img, stats = F.pathtrace(ctx, b, len(f), 2, width=W, height=H, spp=spp, max_depth=1, **cam)
    ctx.sync()
    ref, rays = oracle.pathtrace(pos, ind, oracle.build_bvh(pos, ind), len(f), 2, (10, 10, 10), (0.7, 0.7, 0.7),
                                 cam["eye"], cam["target"], cam["up"], cam["fov_deg"], W, H, spp, 1)
    assert stats["shadow_rays"] == rays[1]
    err = np.abs(img.cpu().numpy() - ref)
    assert (err <= 1e-4 * np.maximum(np.abs(ref), 1.0)).mean() > 0.995
