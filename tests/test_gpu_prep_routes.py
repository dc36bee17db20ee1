"""The preparation's routes by table size (up to 32 patches, up to 512, more):
the same forward and gradient against the FP64 oracle at the paths' bounds on
either side of each limit, and the same refusals."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err
from test_gpu_adjoint import _check, _upstream, run_adjoint

pytestmark = pytest.mark.gpu


def _table(n, seed, hi=14):
    from wave_tool_gb300 import workloads
    w = workloads.small_random(seed, n_patches=n, side_range=(2, 40), n_waves_range=(hi // 20, hi), heightmap=False)
    p = w.patches
    for i in range(0, n, 2):  # every other patch a rectangle, the rest skewed
        p["br"][i][1], p["tl"][i][0] = p["bl"][i][1], p["bl"][i][0]
        p["tr"][i] = p["br"][i][0], p["tl"][i][1]
    return w


# (32 patches of up to 90 waves: more than 1024 pairs)
@pytest.mark.parametrize("n,hi", [(3, 14), (31, 14), (32, 14), (32, 90), (33, 14), (64, 14), (511, 14), (512, 14), (513, 14)])
def test_forward_and_refusals(wt, oracle, gpu, n, hi):
    import torch
    w = _table(n, 5 + n, hi)
    surf = wt.Surface(w.patches, w.waves)
    pos, nrm = surf.displace(flags=wt.WT_OUT_DISPLACEMENT)
    torch.cuda.synchronize()
    assert surf.status()[0] == 0
    _, disp64, _, _ = oracle.displace_f64(w.patches, w.waves)
    assert rel_err(pos[:, :3].double().cpu().numpy(), disp64) <= 1e-5
    # a patch of one column and a wave without a length: reported, the others run
    patches, waves = w.patches.copy(), w.waves.copy()
    one = n // 2
    patches["cols"][one] = 1
    has = [i for i in range(n) if i != one and patches["wave_count"][i] > 0]
    lost = has[-1]
    waves["wavelength"][int(patches["wave_offset"][lost])] = 0.0
    uses = {i for i in range(n) if patches["wave_offset"][i] <= patches["wave_offset"][lost] <
            patches["wave_offset"][i] + patches["wave_count"][i]}
    bad = wt.Surface(w.patches, waves)
    bad.patches.copy_(wt.to_device(patches))
    p2, n2 = bad.displace(torch.zeros_like(pos), torch.zeros_like(nrm), flags=wt.WT_OUT_DISPLACEMENT)
    torch.cuda.synchronize()
    st, at = bad.status()
    assert st != 0 and at == min(uses | {one})
    for i in set(range(n)) - uses - {one}:
        o, k = int(w.patches["out_offset"][i]), int(w.patches["cols"][i]) * int(w.patches["rows"][i])
        assert torch.equal(p2[o:o + k], pos[o:o + k]) and torch.equal(n2[o:o + k], nrm[o:o + k])


@pytest.mark.parametrize("n,hi", [(32, 14), (32, 90), (33, 14), (512, 14), (513, 14)])
@pytest.mark.parametrize("saved", [False, True])
def test_gradient(wt, oracle, gpu, n, hi, saved):
    w = _table(n, 70 + n, hi)
    gp, gn = _upstream(w.n_vertices, n)
    g, _ = run_adjoint(wt, w, gp, gn, saved=saved)
    _check(g, oracle.adjoint_f64(w.patches, w.waves, gp.numpy(), gn.numpy()))
