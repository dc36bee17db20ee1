"""Tables whose matrix-product items do not fill the SMs' rounds evenly (40
column blocks of 200 rows on 152 SMs): the number of rows per item is then
compared with others, in each of the preparation's routes.  The saving forward
against the plain one bit for bit, gradients against the FP64 reference, and the
time against a table whose items fill one round."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from test_gpu_adjoint import _check, _upstream, run_adjoint
from test_gpu_prep_shared import _graph_us

pytestmark = pytest.mark.gpu


def _table(n, cols, rows, k, pool=0, seed=3):
    from wave_tool_gb300 import abi, workloads
    rng = workloads.SplitMix64(seed)
    hx, hz = 0.1 * (cols - 1), 0.1 * (rows - 1)
    patches = np.array([((300.0 * i - hx, hz), (300.0 * i + hx, hz), (300.0 * i - hx, -hz), (300.0 * i + hx, -hz), cols, rows,
                         i * k, k, rng.uniform(0.0, 1e3), 0.0, 0, i * cols * rows) for i in range(n)], dtype=abi.PATCH_DTYPE)
    waves = [w for _ in range(n) for w in workloads.waves_wide(rng, k)] + workloads.waves_wide(rng, max(pool, 1))
    return SimpleNamespace(patches=patches, waves=np.array(waves, dtype=abi.WAVE_DTYPE), heightmap=None,
                           n_vertices=n * cols * rows)


# (20: the route of up to 32 patches; 40; 40 in a pool too large for its bitmask)
@pytest.mark.parametrize("n,cols,rows,pool", [(20, 130, 300, 0), (40, 129, 130, 0), (40, 129, 130, 17000)])
def test_saving_forward_and_gradient(wt, oracle, gpu, n, cols, rows, pool):
    import torch
    w = _table(n, cols, rows, 8, pool)
    surf = wt.Surface(w.patches, w.waves)
    pos, nrm = surf.displace(flags=1)
    sums = torch.zeros((surf.n_vertices, 8), device="cuda")
    p1, n1 = surf.displace(flags=1, sums=sums)
    assert surf.status()[0] == 0
    assert torch.equal(p1, pos) and torch.equal(n1, nrm) and torch.equal(sums[:, :3], pos[:, :3])
    gp, gn = _upstream(w.n_vertices, 5)
    used = slice(0, 8 * n)
    g64 = oracle.adjoint_f64(w.patches, w.waves, gp.numpy(), gn.numpy())
    for saved in (False, True):
        g, _ = run_adjoint(wt, w, gp, gn, saved=saved)
        _check(g, g64, used=used)


def test_an_uneven_table_is_not_much_slower(wt, gpu):
    """40 patches of 129 x 200 against 38 (152 items): the saving forward took 1.5
    times as long."""
    import torch
    us = []
    for n in (40, 38):
        w = _table(n, 129, 200, 8)
        surf = wt.Surface(w.patches, w.waves)
        pos, nrm = surf.alloc_outputs(0)
        sums = torch.empty((surf.n_vertices, 8), device="cuda")
        us.append(_graph_us(lambda: surf.displace(pos, nrm, sums=sums), n=5))
    assert us[0] <= 1.25 * us[1], us


@pytest.mark.parametrize("sizes", [[(503, 503, 9), (40, 40, 50), (123, 123, 25), (130, 131, 14), (114, 114, 36)],
                                   [(700, 100, 8)] * 12])
def test_patches_of_different_sizes(wt, oracle, gpu, sizes):
    """Gradients where the number of items per SM is chosen for patches unlike one
    another, and where the choices come out alike."""
    parts = [_table(1, c, r, k, seed=5 + i) for i, (c, r, k) in enumerate(sizes)]
    patches, waves, v = [], [], 0
    for t in parts:
        p = t.patches.copy()
        p["wave_offset"], p["out_offset"] = len(waves), v
        patches.append(p)
        waves.extend(t.waves)
        v += t.n_vertices
    w = SimpleNamespace(patches=np.concatenate(patches), waves=np.array(waves, dtype=parts[0].waves.dtype), heightmap=None,
                        n_vertices=v)
    gp, gn = _upstream(v, 6)
    g64 = oracle.adjoint_f64(w.patches, w.waves, gp.numpy(), gn.numpy())
    for saved in (False, True):
        g, _ = run_adjoint(wt, w, gp, gn, saved=saved)
        for p in w.patches:
            at = slice(int(p["wave_offset"]), int(p["wave_offset"]) + int(p["wave_count"]))
            _check(g[at], g64[at])
