"""The adjoint's matrix-product path (parallelogram patches of 8 to 64 waves) at
the edges of its tiles (128 columns by 16 rows, half tiles of 8, 32 waves a
step), against the FP64 reference gradient at the path's bound: per field,
|g - g_64| <= 1e-4 of the field's largest |g_64|."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from test_gpu_adjoint import _check, _upstream, run_adjoint
from test_gpu_products import patch_table

pytestmark = pytest.mark.gpu

# each table also holds a skewed patch and one of four waves (the recurrence)
SIZES = [[(32, 2, 8), (33, 7, 9), (127, 8, 31), (128, 9, 32), (300, 64, 40)],
         [(129, 15, 33), (257, 16, 48), (300, 17, 49), (64, 33, 64)],
         [(160, 97, 17), (385, 31, 63), (96, 130, 64), (200, 40, 65), (1030, 5, 24)]]


def _table(sizes, seed, wrap, tex):
    patches, waves, hm = patch_table(sizes, seed, wrap, tex)
    n = int(patches["out_offset"][-1]) + int(patches["cols"][-1]) * int(patches["rows"][-1])
    return SimpleNamespace(patches=patches, waves=waves, heightmap=hm, n_vertices=n)


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("wrap,tex,saved,nrm", [(0, None, False, True), (0, None, True, False), (1, (32, 32), True, True),
                                                (0, (37, 21), False, True)])
def test_products_against_oracle(wt, oracle, gpu, sizes, wrap, tex, saved, nrm):
    w = _table(sizes, 57 + len(sizes) + wrap, wrap, tex)
    gp, gn = _upstream(w.n_vertices, 4)
    gn = gn if nrm else None
    g, texels = run_adjoint(wt, w, gp, gn, saved=saved, oracle=oracle)
    g64 = oracle.adjoint_f64(w.patches, w.waves, gp.numpy(), None if gn is None else gn.numpy(), texels, w.heightmap)
    for p in w.patches:  # each patch has waves of its own
        at = slice(int(p["wave_offset"]), int(p["wave_offset"]) + int(p["wave_count"]))
        _check(g[at], g64[at])


def test_layouts_and_alignment(wt, gpu):
    """float3 gradients and float4 ones off a 16-byte boundary give the same bits."""
    import torch
    w = _table(SIZES[1], 71, 0, None)
    gp, gn = (x.cuda() for x in _upstream(w.n_vertices, 9))
    surf = wt.Surface(w.patches, w.waves)
    want = surf.adjoint(gp, gn).clone()

    def off(x):
        b = torch.empty(x.numel() + 1, device="cuda")
        b[1:].copy_(x.reshape(-1))
        return b[1:].view(x.shape)

    assert torch.equal(surf.adjoint(off(gp), off(gn)), want)
    g3 = surf.adjoint(gp[:, :3].contiguous(), gn[:, :3].contiguous(), flags=wt.WT_LAYOUT_VEC3)
    assert torch.equal(g3, want)


def test_sums_keep_their_own_digits(wt, oracle, gpu):
    """The steepness gradient follows from the horizontal displacement alone: it
    keeps its digits beside vertical gradients 10^9 times as large."""
    w = _table(SIZES[2], 83, 0, None)
    gp, _ = _upstream(w.n_vertices, 2)
    gp[:, 0] *= 1e-9
    gp[:, 2] *= 1e-9
    g64 = oracle.adjoint_f64(w.patches, w.waves, gp.numpy(), None)
    g, _ = run_adjoint(wt, w, gp, None)
    for p in w.patches:
        at = slice(int(p["wave_offset"]), int(p["wave_offset"]) + int(p["wave_count"]))
        scale = np.abs(g64[at, 3]).max()
        assert np.abs(g[at, 3].astype(np.float64) - g64[at, 3]).max() <= 1e-4 * scale


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_that_are_not_finite_stay_visible(wt, gpu, value):
    """One in the upstream gradient of a patch reaches every gradient of its waves
    and no other patch's."""
    w = _table(SIZES[2], 83, 0, None)
    gp, gn = _upstream(w.n_vertices, 2)
    want, _ = run_adjoint(wt, w, gp, gn)
    hit = w.patches[1]
    gp[int(hit["out_offset"]) + 7, 0] = value
    g, _ = run_adjoint(wt, w, gp, gn)
    for p in w.patches:
        at = slice(int(p["wave_offset"]), int(p["wave_offset"]) + int(p["wave_count"]))
        if p["out_offset"] == hit["out_offset"]:
            assert not np.isfinite(g[at]).any()
        else:
            assert np.array_equal(g[at], want[at])
