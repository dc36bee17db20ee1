"""Which patches the adjoint runs as matrix products: tables on either side of
the rule on waves, column blocks and tiles (all products, none, some of them),
from saved sums and recomputing, against the FP64 reference gradient; and a table
of part-filled column blocks is not slower for being parallelograms."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from test_gpu_adjoint import _check, _upstream, run_adjoint
from test_gpu_prep_shared import _graph_us
from test_gpu_uneven_items import _table

pytestmark = pytest.mark.gpu


def _join(*tables):
    patches, waves, v = [], [], 0
    for t in tables:
        p = t.patches.copy()
        p["wave_offset"] += len(waves)
        p["out_offset"] += v
        patches.append(p)
        waves.extend(t.waves)
        v += t.n_vertices
    return SimpleNamespace(patches=np.concatenate(patches), waves=np.array(waves, dtype=tables[0].waves.dtype),
                           heightmap=None, n_vertices=v)


@pytest.mark.parametrize("saved", [False, True])
@pytest.mark.parametrize("parts", [[(40, 129, 130, 40)], [(50, 64, 130, 12), (3, 257, 90, 40), (2, 40, 50, 64)],
                                   [(45, 130, 230, 10), (2, 256, 60, 30)], [(1, 300, 2000, 9), (34, 100, 120, 8)]])
def test_either_side(wt, oracle, gpu, parts, saved):
    w = _join(*[_table(*p, seed=3 + i) for i, p in enumerate(parts)])
    gp, gn = _upstream(w.n_vertices, 6)
    g, _ = run_adjoint(wt, w, gp, gn, saved=saved)
    g64 = oracle.adjoint_f64(w.patches, w.waves, gp.numpy(), gn.numpy())
    for p in w.patches:  # each patch has waves of its own
        at = slice(int(p["wave_offset"]), int(p["wave_offset"]) + int(p["wave_count"]))
        _check(g[at], g64[at])


@pytest.mark.parametrize("saved", [False, True])
def test_part_filled_blocks_are_not_slower(wt, gpu, saved):
    """40 patches of 129 x 200 with 12 waves and the same with a corner moved, which
    the recurrence takes (the products took 1.4 to 1.7 times as long)."""
    import torch
    us = []
    for skew in (False, True):
        w = _table(40, 129, 200, 12)
        if skew:
            w.patches["tr"][:, 0] += 0.25
        surf = wt.Surface(w.patches, w.waves)
        gp, gn = (u.cuda() for u in _upstream(w.n_vertices, 5))
        sums = None
        if saved:
            sums = torch.empty((surf.n_vertices, 8), device="cuda")
            surf.displace(sums=sums)
        g = torch.empty((surf.n_waves, 8), device="cuda")
        us.append(_graph_us(lambda: surf.adjoint(gp, gn, grad=g, sums=sums), n=5))
    assert us[0] <= 1.2 * us[1], us


def test_a_mixed_table_is_one_kernel_s(wt, gpu):
    """30 patches of 8 waves and 10 of 64 against 40 of 64, which the products take as
    long for (split between recurrence and products the mixed table took 1.03 times as
    long, as a whole 0.83)."""
    import torch

    def us(w):
        surf = wt.Surface(w.patches, w.waves)
        gp, gn = (u.cuda() for u in _upstream(w.n_vertices, 5))
        g = torch.empty((surf.n_waves, 8), device="cuda")
        return _graph_us(lambda: surf.adjoint(gp, gn, grad=g), n=5)

    few, many = _table(30, 520, 200, 8), _table(10, 520, 200, 64, seed=4)
    assert us(_join(few, many)) <= 0.95 * us(_table(40, 520, 200, 64))
