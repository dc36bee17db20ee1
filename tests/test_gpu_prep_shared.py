"""Tables whose patches share waves, or use a part of a pool: the preparation's
routes for them against the FP64 oracle on either side of their limits, the same
refusals (a wave that is not valid counts where a patch uses it), waves off a
16-byte boundary, and no route much slower than the same patches with waves of
their own."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err
from test_gpu_adjoint import _check, _upstream, run_adjoint

pytestmark = pytest.mark.gpu


def _table(n, shared=0, own=0, pool=0, side=(2, 30), seed=1):
    """n patches, every other one a rectangle: all with the `shared` waves, or `own`
    each, out of as many waves and `pool` more (behind them, or spread between them)."""
    from wave_tool_gb300 import workloads
    w = workloads.small_random(seed + n, n_patches=n, side_range=side, n_waves_range=(1, 1), heightmap=False)
    p = w.patches
    rng = workloads.SplitMix64(seed + 7 * n)
    for i in range(0, n, 2):
        p["br"][i][1], p["tl"][i][0] = p["bl"][i][1], p["bl"][i][0]
        p["tr"][i] = p["br"][i][0], p["tl"][i][1]
    waves = np.array(workloads.waves_wide(rng, (shared or n * own) + pool), dtype=w.waves.dtype)
    p["wave_count"] = shared or own
    gap = pool // n if own else 0
    p["wave_offset"] = 0 if shared else np.arange(n) * (own + gap)
    w.waves = waves
    return w


ROUTES = [dict(n=33, shared=9), dict(n=64, shared=16), dict(n=256, shared=4), dict(n=1024, shared=12),
          dict(n=1025, shared=12, side=(2, 9)), dict(n=600, own=17, side=(2, 16)),
          dict(n=3, own=10, pool=5000), dict(n=2, shared=600, pool=9000, side=(20, 30)), dict(n=33, own=9, pool=16000),
          dict(n=300, own=9, pool=9000, side=(2, 20)), dict(n=40, own=30, pool=200), dict(n=65, own=4, pool=2100)]


@pytest.mark.parametrize("kw", ROUTES, ids=lambda k: "-".join(f"{a}{b}" for a, b in k.items() if a != "side"))
def test_forward_and_refusals(wt, oracle, gpu, kw):
    import torch
    w = _table(**kw)
    n = len(w.patches)
    surf = wt.Surface(w.patches, w.waves)
    pos, nrm = surf.displace(flags=1)
    torch.cuda.synchronize()
    assert surf.status()[0] == 0
    _, disp64, _, _ = oracle.displace_f64(w.patches, w.waves)
    assert rel_err(pos[:, :3].double().cpu().numpy(), disp64) <= 1e-5
    # the waves off a 16-byte boundary: the same bits
    raw = torch.zeros(surf.waves.numel() + 16, dtype=torch.uint8, device="cuda")
    raw[4:4 + surf.waves.numel()].copy_(surf.waves)
    off = wt.Surface(w.patches, w.waves)
    off.waves = raw[4:4 + surf.waves.numel()]
    p1, n1 = off.displace(flags=1)
    assert torch.equal(p1, pos) and torch.equal(n1, nrm)
    # a wave that no patch uses is not looked at
    used = np.zeros(len(w.waves), bool)
    for p in w.patches:
        used[int(p["wave_offset"]):int(p["wave_offset"]) + int(p["wave_count"])] = True
    if not used.all():
        waves = w.waves.copy()
        waves["wavelength"][np.nonzero(~used)[0][0]] = -1.0
        s = wt.Surface(w.patches, waves)
        p1, n1 = s.displace(flags=1)
        assert s.status()[0] == 0 and torch.equal(p1, pos) and torch.equal(n1, nrm)
    # one that some use, and one that leaves the products no room
    waves = w.waves.copy()
    last = int(w.patches["wave_offset"][n - 1]) + int(w.patches["wave_count"][n - 1]) - 1
    waves["wavelength"][last] = np.nan
    waves["amplitude"][int(w.patches["wave_offset"][0])] = 2.0e12
    waves["steepness_q"][int(w.patches["wave_offset"][0])] = 0.0
    s = wt.Surface(w.patches, waves)
    p2, _ = s.displace(torch.full_like(pos, 7.0), torch.full_like(nrm, 7.0), flags=1)
    hit = [i for i in range(n) if w.patches["wave_offset"][i] <= last < w.patches["wave_offset"][i] + w.patches["wave_count"][i]]
    st, at = s.status()
    assert st == wt.abi.WT_ERR_INVALID_ARG and at == hit[0]
    for i in range(n):
        o, k = int(w.patches["out_offset"][i]), int(w.patches["cols"][i]) * int(w.patches["rows"][i])
        if i in hit:
            assert bool((p2[o:o + k] == 7.0).all())
        elif w.patches["wave_offset"][i] > w.patches["wave_offset"][0]:
            assert torch.equal(p2[o:o + k], pos[o:o + k])


@pytest.mark.parametrize("kw", [ROUTES[1], ROUTES[3], ROUTES[8], ROUTES[9]],
                         ids=lambda k: "-".join(f"{a}{b}" for a, b in k.items() if a != "side"))
def test_gradient(wt, oracle, gpu, kw):
    w = _table(**kw)
    gp, gn = _upstream(w.n_vertices, 3)
    g, _ = run_adjoint(wt, w, gp, gn)
    _check(g, oracle.adjoint_f64(w.patches, w.waves, gp.numpy(), gn.numpy()))


def _graph_us(f, n=20):
    import torch
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        for _ in range(3):
            f()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for _ in range(n):
            f()
    best = 1e9
    for _ in range(20):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        g.replay()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / n * 1e3)
    return best


@pytest.mark.parametrize("kw,same", [(dict(n=64, shared=16), dict(n=64, own=16)),
                                     (dict(n=256, shared=4), dict(n=256, own=4)),
                                     (dict(n=33, own=4, pool=16000), dict(n=33, own=4)),
                                     (dict(n=2, shared=600, pool=60000), dict(n=2, shared=600))])
def test_no_route_is_much_slower(wt, gpu, kw, same):
    """Shared waves, or a pool around the waves that are used, cost at most half as
    much again as waves of their own (they took 1.5 to 3 times as long when one
    block formed all constants, or read the whole pool)."""
    us = []
    for k in (kw, same):
        w = _table(**k, side=(20, 30))
        surf = wt.Surface(w.patches, w.waves)
        pos, nrm = surf.alloc_outputs(0)
        us.append(_graph_us(lambda: surf.displace(pos, nrm)))
    assert us[0] <= 1.5 * us[1], us


def test_a_kernel_that_finds_nothing_costs_little(wt, gpu):
    """The saving forward of 4000 patches of seven waves out of seven, and out of nine
    (with eight the matrix products' kernel runs, and finds no patch): it took 1.06
    times as long when that kernel came first."""
    import torch
    us = []
    for pool in (2, 0):
        w = _table(n=4000, shared=7, pool=pool, side=(24, 25))
        w.waves = w.waves[:7 + pool]
        surf = wt.Surface(w.patches, w.waves)
        pos, nrm = surf.alloc_outputs(0)
        sums = torch.empty((surf.n_vertices, 8), device="cuda")
        us.append(_graph_us(lambda: surf.displace(pos, nrm, sums=sums), n=5))
    assert us[0] <= 1.035 * us[1], us
