"""The waits inside the matrix-product kernels are bounded.  With the limit
shortened for this thread's launches: a call comes back, says WT_ERR_TIMEOUT or
has the usual bits, and leaves nothing behind: the next call with the usual
limit gives the usual bits.  (A limit of 0 has run out from the start.)"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_gpu_adjoint import _upstream
from test_gpu_products import patch_table

pytestmark = pytest.mark.gpu

USUAL = 2_000_000_000


@pytest.fixture
def limit(wt, gpu):
    f = wt.lib().wt_internal_wait_limit
    f.argtypes, f.restype = [C.c_ulonglong], None
    yield f
    f(USUAL)


def _call(wt, surf, what, ups):
    """One call's outputs and status (the outputs start as zeros)."""
    import torch
    if what == "forward":
        pos, nrm = (torch.zeros((surf.n_vertices, 4), device="cuda") for _ in range(2))
        surf.displace(pos, nrm, flags=1)
        return (pos, nrm), surf.status()[0]
    sums = None
    if what == "saved":
        sums = ups[2]
    g = surf.adjoint(ups[0], ups[1], sums=sums)
    return (g,), wt.workspace_status(surf.adj_workspace)[0]


@pytest.mark.parametrize("what", ["forward", "adjoint", "saved"])
@pytest.mark.parametrize("sizes,alone", [([(300, 70, 30)], True), ([(300, 70, 128)], True),
                                         ([(300, 70, 30), (640, 300, 64), (1030, 5, 24)], False)])
def test_a_wait_that_runs_out(wt, gpu, limit, what, sizes, alone):
    import torch
    patches, waves, _ = patch_table(sizes, 41, 0, None)
    if alone:
        patches = patches[:1].copy()
        waves = waves[:sizes[0][2]].copy()
    surf = wt.Surface(patches, waves)
    gp, gn = (u.cuda() for u in _upstream(surf.n_vertices, 3))
    sums = torch.empty((surf.n_vertices, 8), device="cuda")
    surf.displace(flags=1, sums=sums)
    ups = (gp, gn, sums)
    want, st = _call(wt, surf, what, ups)
    assert st == wt.abi.WT_OK
    products = what == "forward" or max(p["wave_count"] for p in patches) <= 64
    for ns in (0, 1, 500, 3000, 20000, USUAL):
        limit(ns)
        got, st = _call(wt, surf, what, ups)
        assert st in (wt.abi.WT_OK, wt.abi.WT_ERR_TIMEOUT)
        if ns == 0 and products:
            assert st == wt.abi.WT_ERR_TIMEOUT
        if st == wt.abi.WT_OK:
            assert all(torch.equal(a, b) for a, b in zip(got, want)), ns
        limit(USUAL)
        got, st = _call(wt, surf, what, ups)
        assert st == wt.abi.WT_OK and all(torch.equal(a, b) for a, b in zip(got, want)), ns


def test_the_limit_is_this_threads(wt, gpu, limit):
    """Another thread's calls keep the usual limit."""
    import threading

    import torch
    patches, waves, _ = patch_table([(300, 70, 30)], 41, 0, None)
    surf = wt.Surface(patches[:1].copy(), np.ascontiguousarray(waves[:30]))
    want, st = _call(wt, surf, "forward", None)
    limit(0)
    out = []
    t = threading.Thread(target=lambda: out.append(_call(wt, surf, "forward", None)))
    t.start()
    t.join()
    assert out[0][1] == wt.abi.WT_OK and all(torch.equal(a, b) for a, b in zip(out[0][0], want))
