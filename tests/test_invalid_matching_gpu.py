"""Arrays that are no matching -- everyone points at a hub, at out of range ids, in
circles, at each other one way -- are reported by the contraction and by the coarse
map, whose arrays they must not lead out of: every vertex that has no partner is
taken as a singleton, so each row is counted once."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _star(leaves):
    n = leaves + 1
    return cm.Graph(np.r_[np.arange(n), n - 1 + leaves], np.r_[np.full(leaves, leaves), np.arange(leaves)])


def _arrays(n, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    m = i ^ 1
    m[m >= n] = i[m >= n]
    some = rng.random(n) < 0.1
    mixed = np.where(some, rng.integers(-5, n + 5, n), m)
    return {"hub": np.full(n, n - 1), "first": np.zeros(n, np.int64), "circle": (i + 1) % n,
            "range": np.where(i % 3 == 0, n + i, np.where(i % 3 == 1, -1 - i, i)), "random": rng.integers(0, n, n),
            "mixed": mixed}


@pytest.mark.parametrize("name", ["hub", "first", "circle", "range", "random", "mixed"])
@pytest.mark.parametrize("graph", ["star", "grid", "rmat"])
def test_no_matching(ctx, graph, name):
    import torch
    g = {"star": lambda: _star(70000), "grid": lambda: cm.gen_grid2d(61, 47),
         "rmat": lambda: cm.gen_rmat(13, 16, seed=2)}[graph]()
    n, d = g.nvtxs, g.to_device()
    bad = _arrays(n, 3)[name].astype(np.int32)
    inside = (bad >= 0) & (bad < n)
    pair = inside & (bad[np.where(inside, bad, 0)] == np.arange(n))
    assert not pair.all()
    t = torch.from_numpy(bad).cuda()
    for call in (ctx.contract, ctx.build_cmap):
        with pytest.raises(cm.CMError) as e:
            call(d, t)
        assert e.value.code == cm.CM_ERR_INVALID
    # what is left in the arrays: the singletons' matching, and the same context goes on
    good = np.where(pair, bad, np.arange(n)).astype(np.int32)
    coarse, cmap, sizes = ctx.contract(d, t, sync=False)
    with pytest.raises(cm.CMError):
        ctx.sync()
    want, wmap = O.contract(O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt), good)
    cn, cm_ = (int(x) for x in sizes.cpu())
    assert (cn, cm_) == (want.n, want.m) and np.array_equal(cmap.cpu().numpy(), wmap)
    for a, b in zip(coarse, (want.xadj, want.adjncy, want.adjwgt, want.vwgt)):
        assert np.array_equal(a.cpu().numpy()[:len(b)], b)
    got, gmap = ctx.contract(d, torch.from_numpy(good).cuda())
    assert np.array_equal(gmap.cpu().numpy(), wmap) and got.nedges == want.m
