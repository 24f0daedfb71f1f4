"""Chains of displaced proposals as long as the graph: a path whose weights grow
along it, or with ties to the lower id one whose vertices are numbered in order,
is settled one step after the other.  Such graphs take their time but are matched,
in every kernel that follows chains: by a lane, by a warp in one pass or in rounds
(where a long chain goes on in the next round), and in the kernel of whole levels,
which hands a long one over."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(n, a, b, w):
    s, d, w = np.r_[a, b], np.r_[b, a], np.r_[w, w]
    order = np.lexsort((d, s))
    return cm.Graph(np.r_[0, np.cumsum(np.bincount(s, minlength=n))], d[order], w[order])


def _path(n, grow=False):
    ends = np.stack([np.arange(n) - 1, np.arange(n) + 1], 1).ravel()
    w = np.stack([np.arange(n), np.arange(n) + 1], 1).ravel() if grow else np.ones(2 * n, np.int32)
    inside = (ends >= 0) & (ends < n)
    return cm.Graph(np.r_[0, 2 * np.arange(1, n) - 1, 2 * n - 2], ends[inside], w[inside])


def _hub_and_path(length, leaves):
    """A path in order, and a hub (the last vertex) whose leaves all prefer
    partners of their own: the hub uses its list up, is scanned by a warp, and
    takes the path's first vertex away from the second."""
    i = np.arange(length - 1)
    leaf = length + np.arange(leaves)
    hub = length + 2 * leaves
    a = np.r_[i, leaf, np.full(leaves, hub), hub]
    b = np.r_[i + 1, leaf + leaves, leaf, 0]
    return _csr(hub + 1, a, b, np.r_[np.ones(length - 1), np.full(leaves, 20), np.full(leaves, 10), 5].astype(np.int64))


@pytest.mark.parametrize("n", [2, 3, 262144, 400001])
def test_path_in_order(ctx, n):
    m, _ = ctx.match(_path(n).to_device(), 100, 0)
    want = np.arange(n) ^ 1
    want[n - n % 2:] = np.arange(n - n % 2, n)
    assert np.array_equal(m.cpu().numpy(), want)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [101, 300000, 8000001])
def test_path_of_growing_weights(ctx, n, mode):
    """The largest is one lane's work for several seconds."""
    m, _ = ctx.match(_path(n, grow=True).to_device(), 100, mode)
    want = n - 1 - (np.arange(n)[::-1] ^ 1)
    if n % 2:
        want[0] = 0
    assert np.array_equal(m.cpu().numpy(), want)


@pytest.mark.parametrize("leaves", [19, 300])
@pytest.mark.parametrize("length", [1000, 300000])
def test_chain_of_a_warp(ctx, length, leaves):
    """One-chunk and several-chunk hubs; the long path spans several rounds."""
    g = _hub_and_path(length, leaves)
    want = O.match_greedy(O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt), 100, 0)
    assert want[0] == g.nvtxs - 1 and want[1] == 2
    m, _ = ctx.match(g.to_device(), 100, 0)
    assert np.array_equal(m.cpu().numpy(), want)


@pytest.mark.parametrize("length", [1000, 150000, 300000])
def test_whole_levels(ctx, length):
    g = _hub_and_path(length, 19)
    hs = []
    for separate in (False, True):
        ctx.set_stage_timing(separate)
        hs.append(ctx.coarsen(g.to_device(), 100, 0, max_levels=2))
    ctx.set_stage_timing(False)
    a, b = hs
    assert a.sizes() == b.sizes()
    for l in range(len(a)):
        x, y = a.copy_level(l), b.copy_level(l)
        for f in ("xadj", "adjncy", "adjwgt", "vwgt"):
            assert np.array_equal(getattr(x[0], f), getattr(y[0], f)), (l, f)
        if x[1] is not None:
            assert np.array_equal(x[1], y[1]) and np.array_equal(x[2], y[2]), l
    a.close()
    b.close()
