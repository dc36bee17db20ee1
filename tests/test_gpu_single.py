"""The one-patch forward kernel against the general path: a one-patch call
gives, bit for bit, what the same patch gives in a table of two, at the edges of
its tiles and wave chunks, in every output mode, and reports what the general
path reports."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def table(cols, rows, n, skew, seed):
    """One patch (cols x rows, n waves) and the same with a second, 2 x 2, one behind it."""
    from wave_tool_gb300 import workloads
    w = workloads.small_random(seed, n_patches=1, side_range=(2, 2), n_waves_range=(1, 1), heightmap=True,
                               wrap=seed % 2, skew=skew)
    rng = workloads.SplitMix64(seed)
    waves = np.array(workloads.waves_wide(rng, n + 1), dtype=w.waves.dtype)
    one = w.patches[:1].copy()
    one["cols"], one["rows"], one["wave_offset"], one["wave_count"] = cols, rows, 1, n
    two = np.concatenate([one, one])
    two["cols"][1] = two["rows"][1] = 2
    two["wave_offset"][1], two["wave_count"][1] = 0, 1
    two["out_offset"][1] = cols * rows
    return one, two, waves, w.heightmap


@pytest.mark.parametrize("cols,rows,n,skew", [(2, 2, 0, True), (31, 5, 1, True), (255, 3, 31, False), (256, 2, 32, True),
                                              (257, 19, 33, True), (513, 40, 64, False), (1024, 9, 127, True),
                                              (33, 700, 5, False)])
@pytest.mark.parametrize("flags", [0, 1, 2, 3])
def test_one_patch_equals_two_patch_table(wt, gpu, cols, rows, n, skew, flags):
    import torch
    one, two, waves, hmw = table(cols, rows, n, skew, cols + n)
    hm = wt.heightmap_from(hmw)
    nv = cols * rows
    a, b = wt.Surface(one, waves, hm), wt.Surface(two, waves, hm)
    pa, na = a.displace(flags=flags)
    pb, nb = b.displace(flags=flags)
    assert torch.equal(pa, pb[:nv]) and torch.equal(na, nb[:nv])
    sa, sb = (torch.zeros((s.n_vertices, 8), device="cuda") for s in (a, b))
    qa, _ = a.displace(flags=flags, sums=sa)
    b.displace(flags=flags, sums=sb)
    assert torch.equal(qa, pa) and torch.equal(sa, sb[:nv])
    assert a.status()[0] == 0 and b.status()[0] == 0
    if not flags & 1:
        cam = wt.camera(position=(0.0, 9.0, 30.0), pitch_deg=-20.0, aspect=1.5, displaceable_amplitude=2.0)
        vd = wt.to_device(wt.projected_grid(cam)[1])
        fa, fb = a.displace_stage(vd), b.displace_stage(vd)
        for k in fa:
            assert torch.equal(fa[k], fb[k][:nv]), k


def test_one_patch_refusals(wt, gpu):
    """A bad corner, a bad wave and a workspace short of wave slots are
    reported as by the general path, and nothing is written."""
    import torch
    one, _, waves, _ = table(40, 30, 40, True, 5)
    cases = []
    p = one.copy(); p["bl"][0, 0] = np.nan
    cases.append((p, waves, wt.abi.WT_ERR_INVALID_ARG))
    w = waves.copy(); w["wavelength"][7] = -1.0
    cases.append((one, w, wt.abi.WT_ERR_INVALID_ARG))
    w = waves.copy(); w["amplitude"][0] = np.inf   # a wave the patch does not use
    cases.append((one, w, wt.abi.WT_OK))
    p = one.copy(); p["wave_count"] = len(waves)   # past the end of the wave array
    cases.append((p, waves, wt.abi.WT_ERR_INVALID_ARG))
    for patches, wv, want in cases:
        s = wt.Surface(patches, wv)
        pos, nrm = torch.full((1200, 4), 7.0, device="cuda"), torch.full((1200, 4), 7.0, device="cuda")
        s.displace(pos, nrm)
        st, bad = s.status()
        assert st == want and (want == wt.abi.WT_OK or bad == 0)
        assert bool((pos == 7.0).all()) == (want != wt.abi.WT_OK)
    s = wt.Surface(one, waves)
    s.workspace = wt.empty_bytes(wt.displace_workspace_bytes(1, 20))
    pos, nrm = torch.full((1200, 4), 7.0, device="cuda"), torch.full((1200, 4), 7.0, device="cuda")
    s.displace(pos, nrm)
    assert s.status()[0] == wt.abi.WT_ERR_NOMEM and bool((pos == 7.0).all())
