"""The shading kernel at viewports that do not fill its tiles (32 x 8 pixels a
block, 8 x 4 a warp), against the oracle within the colours' bound
2e-5 (1 + |c|); textures of every byte value.  The rasteriser's ways of sharing
out a triangle by the size of its box, bit for bit against the oracle."""
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


# boxes in pixels around the limits: a thread's own (24), a warp's rows (2048), 32-bit
# edge functions (117 wide or high), a block's rows of 32 and more and narrower ones
BOXES = [(4, 6), (5, 5), (24, 1), (1, 25), (45, 45), (46, 45), (64, 33), (116, 18), (118, 18), (17, 118), (117, 117),
         (130, 20), (20, 130), (31, 150), (33, 150), (250, 180), (319, 2), (2, 199), (400, 300), (3000, 40)]


@pytest.mark.parametrize("copies", [1, 60])
def test_raster_box_sizes(wt, oracle, gpu, copies):
    import torch
    W, H = 320, 200
    rng = np.random.default_rng(copies)
    verts, tris = [], []
    for w, h in BOXES * copies:
        x0, y0 = rng.uniform(0.0, W) - 0.5 * w, rng.uniform(0.0, H) - 0.5 * h
        # two corners of the box and a third point on its opposite sides
        pts = [(x0, y0 + h * rng.uniform()), (x0 + w * rng.uniform(), y0), (x0 + w, y0 + h)]
        base = len(verts)
        for x, y in pts:
            verts.append((2 * x / W - 1, 2 * y / H - 1, rng.uniform(-0.9, 0.9), 1.0))
        tris.append((base, base + 1, base + 2) if rng.uniform() < 0.5 else (base, base + 2, base + 1))
    verts.append((0.0, 0.0, 0.0, -1.0))  # behind the eye: the last triangle is clipped
    tris.append((0, 1, len(verts) - 1))
    clip, idx = np.asarray(verts, np.float32), np.asarray(tris, np.uint32)
    got = wt.water_raster(torch.from_numpy(clip).cuda(), torch.from_numpy(idx.view(np.int32).ravel()).cuda(), W, H)
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy().view(np.uint64).ravel(), oracle.water_raster(clip, idx.ravel(), W, H))


def test_raster_queue_of_several_rounds(wt, oracle, gpu):
    """More queued triangles than the second pass takes in one round."""
    import torch
    W, H, n = 320, 200, 160_000
    rng = np.random.default_rng(7)
    p = rng.uniform(-1.0, 1.0, (n, 1, 2)) + rng.uniform(0.0, 1.0, (n, 3, 2)) * np.array([16 / W, 16 / H])
    clip = np.concatenate([p, rng.uniform(-0.9, 0.9, (n, 3, 1)), np.ones((n, 3, 1))], 2).reshape(-1, 4).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.uint32)
    got = wt.water_raster(torch.from_numpy(clip).cuda(), torch.from_numpy(idx.view(np.int32)).cuda(), W, H)
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy().view(np.uint64).ravel(), oracle.water_raster(clip, idx, W, H))
