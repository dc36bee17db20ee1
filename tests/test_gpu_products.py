"""The forward's matrix-product path (parallelogram patches of 8 to 128 waves)
at the edges of its tiles (128 columns by 32 or 16 rows, 32 waves a step, two
accumulators above 48 waves), against the FP64 oracle at the path's bounds, and
one patch alone against the same patch in a table, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import angle_deg, rel_err

pytestmark = pytest.mark.gpu


def patch_table(sizes, seed, wrap, tex):
    """Parallelogram patches (cols, rows, waves), a skewed one and one of four waves."""
    from wave_tool_gb300 import workloads
    rng = workloads.SplitMix64(seed)
    base = workloads.small_random(seed, n_patches=1, side_range=(40, 40), n_waves_range=(9, 9), heightmap=True, wrap=wrap)
    rows, waves, out = [], [], 0
    for cols, rws, n in [*sizes, (40, 40, 9), (50, 21, 4)]:
        if (cols, rws, n) == (40, 40, 9):
            p = base.patches.copy()
        else:
            hx, hz = 0.185 * (cols - 1), 0.185 * (rws - 1)
            cx, cz = rng.uniform(-2000, 2000), rng.uniform(-2000, 2000)
            s = 0.25 * hx  # a sheared parallelogram: exact in FP32 when the shear is one float
            p = base.patches.copy()
            f = np.float32
            bl, e1, e2 = np.array([f(cx - hx), f(cz + hz)]), np.array([f(2 * hx), f(0)]), np.array([f(s), f(-2 * hz)])
            for k, v in (("bl", bl), ("br", bl + e1), ("tl", bl + e2)):
                p[k] = v
            p["tr"] = p["br"].astype(np.float64) + p["tl"] - p["bl"]
            exact = np.all(p["tr"].astype(np.float64) - p["tl"] - p["br"] + p["bl"] == 0)
            if not exact:  # fall back to an axis-aligned one, exact by construction
                p["bl"], p["br"], p["tl"], p["tr"] = (cx - hx, cz + hz), (cx + hx, cz + hz), (cx - hx, cz - hz), (cx + hx, cz - hz)
            p["cols"], p["rows"] = cols, rws
            p["time_s"] = rng.uniform(0.0, 5.0e3)
        p["wave_offset"], p["wave_count"], p["out_offset"] = len(waves), n, out
        rows.append(p)
        waves.extend(workloads.waves_wide(rng, n))
        out += cols * rws
    hm = workloads.Heightmap(*tex, 0.05, 0.3, wrap, workloads.noise_terms(rng, n=8, kmax=3)) if tex else None
    return np.concatenate(rows), np.array(waves, dtype=base.waves.dtype), hm


SIZES = [[(32, 2, 8), (33, 15, 9), (127, 16, 31), (128, 17, 32)],
         [(129, 31, 33), (257, 32, 48), (300, 33, 49), (64, 65, 64)],
         [(160, 97, 65), (385, 18, 127), (96, 130, 128), (1030, 5, 24)]]


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("wrap,tex,flags", [(0, None, 1), (0, (32, 16), 3), (1, (37, 21), 1), (1, (32, 32), 0)])
def test_products_against_oracle(wt, oracle, gpu, sizes, wrap, tex, flags):
    import torch
    patches, waves, hmw = patch_table(sizes, 31 + len(sizes) + wrap, wrap, tex)
    hm = wt.heightmap_from(hmw)
    surf = wt.Surface(patches, waves, hm)
    pos, nrm = surf.displace(flags=flags)
    torch.cuda.synchronize()
    assert surf.status()[0] == 0
    texels = hm.texels.cpu().numpy() if hm is not None else None
    pos64, disp64, nrm64, edge = oracle.displace_f64(patches, waves, texels, hmw)
    want = disp64 if flags & 1 else pos64
    got = pos[:, :3].double().cpu().numpy()
    assert rel_err(got, want) <= 1e-5
    ok = edge > 1e-3
    assert angle_deg(nrm[:, :3].double().cpu().numpy()[ok], nrm64[ok]).max() < 1e-2
    # each patch alone: the same bits
    for p in patches:
        one = p.reshape(1).copy()
        o, n = int(one["out_offset"][0]), int(one["cols"][0]) * int(one["rows"][0])
        one["out_offset"] = 0
        a = wt.Surface(one, waves[int(p["wave_offset"]):int(p["wave_offset"]) + int(p["wave_count"])].copy(), hm)
        a.host_patches["wave_offset"] = 0
        a.patches.copy_(wt.to_device(a.host_patches))
        p1, n1 = a.displace(flags=flags)
        assert torch.equal(p1, pos[o:o + n]) and torch.equal(n1, nrm[o:o + n])


def test_waves_out_of_the_products_range(wt, oracle, gpu):
    """Waves whose coefficients leave the products' common scale no room, and
    patches of no amplitude, give finite results as before."""
    import torch
    patches, waves, _ = patch_table([(130, 20, 10), (64, 40, 12)], 5, 0, None)
    waves["amplitude"][3] = 2e12
    waves["steepness_q"][3] = 0.0
    waves["amplitude"][10:22] = 0.0
    for table in (patches, patches[1:2].copy()):
        table = table.copy()
        table["out_offset"] -= table["out_offset"][0]
        surf = wt.Surface(table, waves)
        pos, nrm = surf.displace(flags=1)
        torch.cuda.synchronize()
        assert surf.status()[0] == 0
        _, disp64, _, _ = oracle.displace_f64(table, waves, None, None)
        assert rel_err(pos[:, :3].double().cpu().numpy(), disp64) <= 1e-5 or np.abs(disp64).max() == 0
        assert bool(torch.isfinite(pos).all()) and bool(torch.isfinite(nrm).all())


# Ten waves of 15 to 60 m, as steep when their lengths are `far` times as large: the
# displacements' coefficients grow with them, the slopes' stay.  A slope sum is
# off by 2^-22 of each coefficient (two halves of 11 bits), 2 x 1e-7 (sines) and
# 2^-23 (two truncated steps), 5.6e-7 times the coefficients' sum (at most 10 x
# 2 pi / 100); the normal's rounding adds 3 x 2^-24: 5.4e-7 rad.
@pytest.mark.parametrize("far", [2.0**0, 2.0**16, 2.0**20, 2.0**26, 2.0**30])
@pytest.mark.parametrize("alone", [True, False])
def test_slopes_beside_large_displacements(wt, oracle, gpu, far, alone):
    import torch
    from wave_tool_gb300 import workloads
    rng = workloads.SplitMix64(77)
    waves = np.array(workloads.waves_wide(rng, 10, lam=(15.0 * far, 60.0 * far)), dtype=wt.WAVE_DTYPE)
    h = 60.0 * far
    one = np.array([((-h, h), (h, h), (-h, -h), (h, -h), 160, 96, 0, 10, 100.0, 0.0, 0, 0)], dtype=wt.PATCH_DTYPE)
    table = one if alone else np.concatenate([one, one])
    table["out_offset"][1:] = 160 * 96
    surf = wt.Surface(table, waves)
    pos, nrm = surf.displace(flags=1)
    torch.cuda.synchronize()
    assert surf.status()[0] == 0
    _, disp64, nrm64, _ = oracle.displace_f64(table, waves, None, None)
    assert rel_err(pos[:, :3].double().cpu().numpy(), disp64) <= 1e-5
    assert np.radians(angle_deg(nrm[:, :3].double().cpu().numpy(), nrm64)).max() <= 5.4e-7


# What the accumulators' truncation takes from the sums on average (a part of
# them), in units of 2^-25: half of the steps' count in any order of the waves is
# given back, rounded to 2^-23 (so to 2 of these units).  Left are, in no order, that rounding and a quarter of the loss;
# with the largest waves first the other half of it too (128 waves: 16 steps).
@pytest.mark.parametrize("n,order,units", [(48, 0, 2 + 6.2 / 4), (64, 0, 2 + 4.5 / 4), (128, 0, 2 + 8.5 / 4),
                                           (128, -1, 2 + 16 - 8.5), (128, 1, 2 + 8.5)])
def test_sums_are_not_short(wt, oracle, gpu, n, order, units):
    import torch
    from wave_tool_gb300 import workloads
    bias = []
    for seed in range(4):
        rng = workloads.SplitMix64(500 + seed)
        waves = np.array(workloads.waves_wide(rng, n), dtype=wt.WAVE_DTYPE)
        if order:
            waves = waves[np.argsort(order * waves["amplitude"])]
        table = np.array([((-70.0, 50.0), (70.0, 50.0), (-70.0, -50.0), (70.0, -50.0), 300, 200, 0, n, 100.0, 0.0, 0, 0)],
                         dtype=wt.PATCH_DTYPE)
        pos, _ = wt.Surface(table, waves).displace(flags=1)
        torch.cuda.synchronize()
        _, disp64, _, _ = oracle.displace_f64(table, waves, None, None)
        bias.append(float(((pos[:, :3].double().cpu().numpy() - disp64) * disp64).sum() / (disp64 * disp64).sum()))
    assert abs(np.mean(bias)) <= units * 2.0**-25


@pytest.mark.parametrize("alone", [True, False])
def test_displacements_of_a_patch_wider_than_float(wt, gpu, alone):
    """The displacement does not depend on where the grid point is: finite on a
    patch whose sides overflow FP32, as large as its waves at most."""
    import torch
    from wave_tool_gb300 import workloads
    waves = np.array(workloads.waves_wide(workloads.SplitMix64(3), 9), dtype=wt.WAVE_DTYPE)
    h = 3.0e38
    one = np.array([((-h, h), (h, h), (-h, -h), (h, -h), 70, 40, 0, 9, 1.0, 0.0, 0, 0)], dtype=wt.PATCH_DTYPE)
    table = one if alone else np.concatenate([one, one])
    table["out_offset"][1:] = 70 * 40
    pos, _ = wt.Surface(table, waves).displace(flags=1)
    assert bool(torch.isfinite(pos).all())
    most = float(np.abs(waves["amplitude"] * np.maximum(1.0, waves["steepness_q"])).sum())
    assert float(pos[:, :3].abs().max()) <= most


@pytest.mark.parametrize("alone", [True, False])
def test_saved_sums_off_a_sector(wt, gpu, alone):
    """The saved sums on a 16-byte boundary that is no 32-byte one: the same bits."""
    import torch
    patches, waves, _ = patch_table(SIZES[0], 47, 0, None)
    if alone:
        patches = patches[3:4].copy()
        patches["out_offset"] = 0
    surf = wt.Surface(patches, waves)
    want = torch.zeros((surf.n_vertices, 8), device="cuda")
    p0, n0 = surf.displace(flags=1, sums=want)
    buf = torch.zeros(8 * surf.n_vertices + 8, device="cuda")
    off = buf[4:4 + 8 * surf.n_vertices].view(-1, 8)
    assert want.data_ptr() % 32 == 0 and off.data_ptr() % 32 == 16
    p1, n1 = surf.displace(flags=1, sums=off)
    assert surf.status()[0] == 0
    assert torch.equal(off, want) and torch.equal(p1, p0) and torch.equal(n1, n0)
    assert bool((buf[:4] == 0).all()) and bool((buf[-4:] == 0).all())


# A normal from the saved sums: 1 - sum, two products and their rounding, the inverse
# root (2 ulp) and the product with it, at most 8 x 2^-24 in all, twice that where the
# cross product's terms add up.
@pytest.mark.parametrize("cols", [32, 33, 64, 65, 95, 96, 97, 128, 129, 160, 223])
@pytest.mark.parametrize("alone", [True, False])
def test_saved_sums_at_every_width(wt, gpu, cols, alone):
    """All eight sums of each vertex in their places, where warps of the epilogue have
    all, some or none of their 32 columns: the displacement's three are the outputs,
    the slopes' five give the normals."""
    import torch
    patches, waves, _ = patch_table([(cols, 21, 9), (cols, 4, 60)], 11, 0, None)
    patches["y_offset"] = 0.0
    if alone:
        patches = patches[:1].copy()
    surf = wt.Surface(patches, waves)
    sums = torch.full((surf.n_vertices + 1, 8), 7.0, device="cuda")
    pos, nrm = surf.displace(flags=1, sums=sums[:-1])
    assert surf.status()[0] == 0
    assert torch.equal(sums[:-1, :3], pos[:, :3]) and bool((sums[-1] == 7.0).all())
    jx, jz, sxx, sxz, szz = (sums[:-1, i].double() for i in (3, 4, 5, 6, 7))
    n = torch.linalg.cross(torch.stack([-sxz, jz, 1 - szz], 1), torch.stack([1 - sxx, jx, -sxz], 1))
    n = n / n.norm(dim=1, keepdim=True)
    assert float((nrm[:, :3].double() - n).abs().max()) <= 2.0**-20
