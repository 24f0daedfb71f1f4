"""Adjacencies with entries that have no counterpart and whose matching takes many
rounds of mutual proposals: the work has to follow the rows looked at, not rounds
times vertices.  Bit-exact against the oracle's rounds, or where those would take
too long against the outcome by hand."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _path_without(n, i):
    """A path in order in which vertex i + 1 lacks its entry for i."""
    row = np.repeat(np.arange(n), 2)
    col = row + np.tile([-1, 1], n)
    keep = (col >= 0) & (col < n) & ~((row == i + 1) & (col == i))
    return cm.Graph(np.r_[0, np.cumsum(np.bincount(row[keep], minlength=n))], col[keep])


def _waiting(k):
    """Pairs (2 j, 2 j + 1); each first vertex would rather have the first of the
    pair before, which has no entry for it: one pair becomes free at a time."""
    xadj, adj, w = [0], [], []
    for j in range(k):
        adj += ([2 * j - 2] if j else []) + [2 * j + 1]
        w += ([5] if j else []) + [1]
        xadj.append(len(adj))
        adj.append(2 * j)
        w.append(1)
        xadj.append(len(adj))
    return cm.Graph(xadj, adj, w)


def _match(ctx, g, mode):
    return ctx.match(g.to_device(), 100, mode)[0].cpu().numpy()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,i", [(3, 0), (3000, 0), (3001, 1), (3001, 1500), (3001, 1501), (3000, 2998)])
def test_path(ctx, n, i, mode):
    g = _path_without(n, i)
    want = O.match_rounds(O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt), 100, mode, n)[0]
    assert np.array_equal(_match(ctx, g, mode), want)


@pytest.mark.parametrize("n", [600001, 800001])  # one block alone, and all of them
def test_long_path(ctx, n):
    i = n // 2 & ~1
    want = np.arange(n) ^ 1
    want[i] = i
    want[i + 1:] = i + 1 + (np.arange(n - i - 1) ^ 1)
    if (n - i - 1) % 2:
        want[-1] = n - 1
    assert np.array_equal(_match(ctx, _path_without(n, i), 0), want)


@pytest.mark.parametrize("mode", [0, 1])
def test_vertices_that_nobody_wakes(ctx, mode):
    g = _waiting(400)
    want = O.match_rounds(O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt), 100, mode, 1000)[0]
    assert np.array_equal(want, np.arange(800) ^ 1)
    assert np.array_equal(_match(ctx, g, mode), want)


@pytest.mark.parametrize("mode", [0, 1])
def test_batch_beside_symmetric_graphs(ctx, mode):
    gs = [cm.gen_grid2d(40, 30), _path_without(501, 200), cm.gen_rmat(9, 8, seed=4), _waiting(50)]
    hs = ctx.coarsen_batch(gs, [1] * len(gs), mode, maxvwgt=100, max_levels=1)
    for g, h in zip(gs, hs):
        want = O.match_rounds(O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt), 100, mode, 2000)[0]
        assert np.array_equal(h.copy_level(0)[2], want)
        h.close()
