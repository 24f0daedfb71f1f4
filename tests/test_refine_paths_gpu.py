"""Refinement passes whose part groups span several blocks' worth of records
and stop at the balance limits, against the sequential model (exact for two
parts), and with more parts the limits themselves."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _refine(ctx, g, k, where):
    import torch
    w = torch.from_numpy(where.copy()).cuda()
    moves = ctx.refine_kway(g.to_device(), k, w)
    return w.cpu().numpy(), moves


def _graph(name, vmax, seed):
    g = {"rmat": lambda: cm.gen_rmat(13, 8, seed=seed), "rgg": lambda: cm.gen_rgg(9000, 40.0, seed=seed),
         "grid": lambda: cm.gen_grid2d(130, 90)}[name]()
    rng = np.random.default_rng(seed)
    return cm.Graph(g.xadj, g.adjncy, g.adjwgt, rng.integers(1, vmax + 1, g.nvtxs))


@pytest.mark.parametrize("name", ["rmat", "rgg", "grid"])
@pytest.mark.parametrize("vmax", [1, 40])
@pytest.mark.parametrize("share", [0.5, 0.48, 0.2])
def test_two_parts_equal_the_sequential_walk(ctx, name, vmax, share):
    """Random parts, balanced, near a limit and far from balance: stretches of
    moves and of refusals, groups of up to thousands of records."""
    g = _graph(name, vmax, 3)
    where = (np.random.default_rng(5).random(g.nvtxs) >= share).astype(np.int32)
    got, moves = _refine(ctx, g, 2, where)
    want = where.copy()
    og = O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt)
    want, wmoves = O.refine_kway_model(og, where, 2)
    np.testing.assert_array_equal(got, want)
    assert moves == wmoves


@pytest.mark.parametrize("k", [3, 16, 200, 1100])
def test_many_parts_keep_the_limits(ctx, k):
    """A part that starts inside its window stays inside it, and every moved
    vertex went to its boundary target."""
    g = _graph("rmat", 3, 7)
    rng = np.random.default_rng(k)
    where = rng.permutation(np.arange(g.nvtxs) % k).astype(np.int32)
    got, moves = _refine(ctx, g, k, where)
    flag, target = O.boundary_targets(O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt), where, k)
    changed = got != where
    assert changed.sum() == moves and flag[changed].all()
    np.testing.assert_array_equal(got[changed], target[changed])
    before, after = (np.bincount(w, weights=g.vwgt, minlength=k) for w in (where, got))
    share = np.float32(np.float32(1.0 / k) * np.float32(g.vwgt.sum()))
    hi, lo = int(share * np.float32(1.03)), int(share / np.float32(1.03))
    inside = (before >= lo) & (before <= hi)
    assert (after[inside] >= lo).all() and (after[inside] <= hi).all()
