"""Refinement with more than two parts, whose groups race: a full part that many
vertices want to enter while several other parts take vertices out of it at the
same time.  Parts that start inside their windows stay inside, at every pass."""
import numpy as np
import pytest

import cumetis_gb300 as cm

pytestmark = pytest.mark.gpu


def _flows(weights, flows, seed):
    """Parts of the given weights (unit vertices).  flows: (from, to, vertices)
    that want to move; each has one edge, to one of two vertices of its target part
    that hold together.  All others have no edges.  -> (graph, partition)"""
    k = len(weights)
    where = np.repeat(np.arange(k), weights)
    np.random.default_rng(seed).shuffle(where)
    members = [np.flatnonzero(where == p) for p in range(k)]
    a, b, w = [m[0] for m in members], [m[1] for m in members], [1 << 20] * k
    used = [2] * k
    src, dst = [np.array(a)], [np.array(b)]
    wgt = [np.array(w)]
    for p, q, count in flows:
        src.append(members[p][used[p]:used[p] + count])
        assert len(src[-1]) == count
        used[p] += count
        dst.append(np.full(count, members[q][0]))
        wgt.append(np.ones(count, np.int64))
    s, d, x = np.concatenate(src), np.concatenate(dst), np.concatenate(wgt)
    s, d, x = np.r_[s, d], np.r_[d, s], np.r_[x, x]
    order = np.lexsort((d, s))
    n = len(where)
    return cm.Graph(np.r_[0, np.cumsum(np.bincount(s, minlength=n))], d[order], x[order]), where.astype(np.int32)


@pytest.mark.parametrize("down", [False, True])
@pytest.mark.parametrize("takers,room", [(8, 800), (30, 600)])
def test_full_part_between_givers_and_takers(ctx, takers, room, down):
    import torch
    share, givers = 20000, 4
    hi, lo = int(np.float32(share) * np.float32(1.03)), int(np.float32(share) / np.float32(1.03))
    k = givers + 1 + takers
    rest = k * share - hi - takers * (hi - room)
    weights = [rest // givers + (i < rest % givers) for i in range(givers)] + [hi] + [hi - room] * takers
    assert sum(weights) == k * share and all(lo <= x <= hi for x in weights)
    flows = [(p, givers, weights[p] - 2) for p in range(givers)]
    flows += [(givers, givers + 1 + t, min(room, (hi - 2) // takers)) for t in range(takers)]
    if down:  # the same towards lower part ids
        flip = lambda p: k - 1 - p
        flows = [(flip(p), flip(q), c) for p, q, c in flows]
        weights = weights[::-1]
    g, where = _flows(weights, flows, takers)
    d = g.to_device()
    for _ in range(30):
        x = torch.from_numpy(where).cuda()
        moves = ctx.refine_kway(d, k, x)
        got = x.cpu().numpy()
        after = np.bincount(got, minlength=k)
        assert moves == (got != where).sum() > 0
        assert after.max() <= hi and after.min() >= lo, after
