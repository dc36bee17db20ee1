"""The shading kernel at viewports that do not fill its tiles (32 x 8 pixels a
block, 8 x 4 a warp), against the oracle within the colours' bound
2e-5 (1 + |c|); textures of every byte value."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_water import CAMERAS, frame, np_, textures

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (8, 4), (7, 3), (31, 9), (32, 8), (33, 17), (129, 65)])
@pytest.mark.parametrize("depth", [False, True])
def test_shade_viewports(wt, oracle, gpu, W, H, depth):
    import torch
    stage, idx = frame(wt, wt.camera(displaceable_amplitude=1.5, **CAMERAS[1]), side=65)
    tx = textures(np.random.default_rng(W + H), W, H)
    if not depth:
        del tx["scene_depth"]
    sh = wt.water_shading(sun_position=(0.6, 0.8, 0.0), fog_colour=(0.8, 0.85, 0.9, 0.3), fog_radius_near=0.01,
                          fog_radius_far=0.2)
    frags = wt.water_raster(stage["clip"], idx, W, H, scene_depth=tx.get("scene_depth"))
    col = wt.water_shade(frags, stage["clip"], idx, stage, W, H, sh, **tx)
    torch.cuda.synchronize()
    shd = {k: getattr(sh, k) for k, _ in sh._fields_}
    shd = {k: (tuple(v) if hasattr(v, "__len__") else v) for k, v in shd.items()}
    U, keep = oracle.frag_uniforms(shd, W, H, **{k: np_(v) for k, v in tx.items()})
    want, _ = oracle.water_shade(frags.cpu().numpy().view(np.uint64).ravel(), np_(stage["clip"]),
                                 np_(idx).view(np.uint32), np_(stage["facing"]), np_(stage["nrm_yaw"]),
                                 np_(stage["view"]), np_(stage["ndc0"]), U)
    assert np.all(np.abs(col.cpu().numpy().reshape(-1, 4) - want) <= 2e-5 * (1.0 + np.abs(want)))
