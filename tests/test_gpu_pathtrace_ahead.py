"""Path tracing with the queue lengths on the device (4-wide handles) against
the same with the host waiting for each of them (any other handle): images bit
for bit and the same ray counts, over paths that end early, passes of one
iteration, batches of samples and renders in a row."""
import numpy as np
import pytest

import gpu_util as U
from fledge_gb300.scenes import icosphere, quad_light

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,spp,depth", [(1, 1, 9, 0), (33, 17, 7, 0), (33, 17, 3, 1), (64, 36, 4, 2), (40, 30, 2, 60)])
def test_images_do_not_depend_on_who_counts(ctx, W, H, spp, depth):
    import fledge_gb300 as F
    v, f = icosphere(3)
    lv, lf = quad_light()
    pos, ind = np.concatenate([v, lv], 0), np.concatenate([f, lf + len(v)], 0)
    cam = dict(eye=(0.0, 0.6, 3.5), target=(0.0, 0.0, 0.0), up=(0.0, 1.0, 0.0), fov_deg=40.0)
    grid = U.dev(np.random.default_rng(3).random((9, 8, 7), dtype=np.float32))
    vol = F.DenseGridVolume(grid, (-1.5,) * 3, (1.5,) * 3, F.Medium(0.8, 0.2, 0.3), ctx)
    out = []
    for width in (4, 8):
        b, _ = U.gpu_build(ctx, pos, ind, width=width)
        for volume in (None, vol):
            for _ in range(2):
                img, st = F.pathtrace(ctx, b, len(f), 2, width=W, height=H, spp=spp, max_depth=depth, volume=volume,
                                      seed=4, **cam)
            ctx.sync()
            out.append((img.cpu().numpy(), st))
    for a, e in zip(out[:2], out[2:]):
        assert np.array_equal(a[0], e[0]) and a[1] == e[1]
        assert a[1]["closest_rays"] >= W * H * spp
