"""Every launch shape the forward kernel supports (and the autotuner may
pick) against the FP64 oracle, through the C ABI: vertices per lane 4 / 8,
8 / 16 / 20 warps per block, register or shared-memory epilogue, wave chunks of
16 and 32.  Shapes with the same vertices per lane tile every patch the same way
and give identical bits."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import angle_deg, rel_err

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 0), (8, 16, 0), (8, 20, 0), (8, 8, 1), (8, 16, 1), (4, 8, 0)]  # (vpl, warps, epi)


@pytest.fixture
def default_tuning(wt):
    yield
    wt.check(wt.lib().wt_set_tuning(None))


def test_every_launch_shape(wt, oracle, gpu, default_tuning):
    import torch
    from wave_tool_gb300 import workloads
    w = workloads.small_random(17, n_patches=6, side_range=(2, 400))
    hm = wt.heightmap_from(w.heightmap)
    surf = wt.Surface(w.patches, w.waves, hm)
    tex = hm.texels.cpu().numpy()
    _, disp64, nrm64, edge = oracle.displace_f64(w.patches, w.waves, tex, w.heightmap)
    ok = edge > 1e-3
    first = {}
    for vpl, warps, epi in SHAPES:
        for chunk in (16, 32):
            wt.set_tuning(warps, 0, chunk, vpl, epi)
            assert wt.get_tuning()["epilogue_in_shared"] == epi
            pos, nrm = surf.displace(flags=wt.WT_OUT_DISPLACEMENT)
            torch.cuda.synchronize()
            assert surf.status()[0] == 0
            p, n = pos.cpu().numpy(), nrm.cpu().numpy()
            assert rel_err(p[:, :3].astype(np.float64), disp64) <= 1e-5, (vpl, warps, epi, chunk)
            assert angle_deg(n[ok, :3].astype(np.float64), nrm64[ok]).max() < 1e-2, (vpl, warps, epi, chunk)
            if vpl in first:
                assert np.array_equal(p, first[vpl][0]) and np.array_equal(n, first[vpl][1]), (vpl, warps, epi,
                                                                                                  chunk)
            else:
                first[vpl] = (p, n)


def test_unsupported_shape_is_rejected(wt, gpu, default_tuning):
    with pytest.raises(wt.WtError):
        wt.set_tuning(16, 0, 32, 4, 1)   # 4 vertices per lane only with 8 warps and the register epilogue
    with pytest.raises(wt.WtError):
        wt.set_tuning(8, 0, 32, 8, 3)
    with pytest.raises(wt.WtError):
        wt.set_tuning(20, 0, 32, 8, 1)   # 20 warps only with the register epilogue


def test_autotune_picks_a_supported_shape(wt, gpu, default_tuning):
    from wave_tool_gb300 import workloads
    w = workloads.config3(n_patches=16, seed=4)
    surf = wt.Surface(w.patches, w.waves, wt.heightmap_from(w.heightmap))
    pos, nrm = surf.alloc_outputs(0)
    best = surf.autotune(pos, nrm, reps=2)
    assert (best["max_vertices_per_lane"], best["warps_per_block"], best["epilogue_in_shared"]) in SHAPES
    assert best["wave_chunk"] in (16, 32)


def _one_launch(wt, surf):
    """Whether a one-patch call runs in the one-patch kernel: the preparation's
    arrays behind the workspace's header stay as they are."""
    import torch
    surf.workspace.fill_(0xAA)
    surf.displace()
    torch.cuda.synchronize()
    assert surf.status()[0] == 0
    return bool((surf.workspace[256:272] == 0xAA).all())


def test_a_table_of_products_has_no_shape_to_tune(wt, gpu, default_tuning):
    """Where no patch runs by the recurrence every shape is the same launch: the
    default stays, for this table and for others of its counts."""
    from wave_tool_gb300 import workloads
    default = wt.get_tuning()
    for n in (16, 1):
        w = workloads.config3(n_patches=n, seed=4)
        w.patches["cols"], w.patches["rows"] = 130, 90
        for i in range(n):
            w.patches["out_offset"][i] = i * 130 * 90
        surf = wt.Surface(w.patches, w.waves)
        pos, nrm = surf.alloc_outputs(0)
        for _ in range(3):
            best = surf.autotune(pos, nrm, reps=1)
            assert {k: best[k] for k in default} == default
    assert _one_launch(wt, surf)


def test_a_large_patch_does_not_tune_a_small_one(wt, gpu, default_tuning):
    """One-patch tables of as many waves: whatever shape a large skewed patch
    gets, a small one runs in the one-patch kernel."""
    import torch
    from wave_tool_gb300 import workloads
    small = workloads.small_random(5, n_patches=1, side_range=(60, 60), n_waves_range=(40, 40), heightmap=False)
    large = small.patches.copy()
    large["cols"] = large["rows"] = 1500
    big = wt.Surface(large, small.waves)
    pos, nrm = big.alloc_outputs(0)
    cam = wt.camera(position=(0.0, 9.0, 30.0), pitch_deg=-20.0, aspect=1.5, displaceable_amplitude=2.0)
    view = wt.to_device(wt.projected_grid(cam)[1])
    best = big.autotune(pos, nrm, reps=2)
    big.autotune_stage(view, big.displace_stage(view), reps=1)
    assert (best["max_vertices_per_lane"], best["warps_per_block"], best["epilogue_in_shared"]) in SHAPES
    torch.cuda.synchronize()
    assert _one_launch(wt, wt.Surface(small.patches, small.waves))


def test_one_patch_of_products_is_tuned_by_route(wt, gpu, default_tuning):
    """A large patch of many waves is faster in the general path's launches than in the
    one-patch kernel: the tuned call takes the faster of the two."""
    import torch
    from wave_tool_gb300 import workloads
    w = workloads.config5(time_s=100.0)
    surf = wt.Surface(w.patches, w.waves)
    pos, nrm = surf.alloc_outputs(0)

    def us():
        best = 1e9
        for _ in range(20):
            pos.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            surf.displace(pos, nrm, flags=0)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        return best

    default = wt.get_tuning()
    one = us()
    wt.set_tuning(16, 0, 32, 8, 0)
    three = us()
    wt.set_tuning(*[default[k] for k in ("warps_per_block", "blocks_per_sm", "wave_chunk", "max_vertices_per_lane",
                                         "epilogue_in_shared")])
    p0, n0 = surf.displace(flags=0)
    surf.autotune(pos, nrm, reps=3)
    tuned = us()
    assert tuned <= 1.04 * min(one, three), (tuned, one, three)
    p1, n1 = surf.displace(flags=0)
    assert torch.equal(p0, p1) and torch.equal(n0, n1)
