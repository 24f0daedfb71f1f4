"""Edges whose two entries differ in weight: the matching is that of mutual
proposals, each vertex going by its own row, also where every proposal ends up
returned.  Bit-exact against the oracle's rounds."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _four():
    """0 and 1 prefer each other, but the offers of 2 and 3 weigh more: (0, 3) and
    (1, 2) end with every offer returned."""
    return cm.Graph([0, 2, 4, 5, 6], [1, 3, 0, 2, 1, 0], [5, 1, 5, 1, 10, 10])


def _changed(g, share, wmax, seed):
    rng = np.random.default_rng(seed)
    w = g.adjwgt.copy()
    some = rng.random(g.nedges) < share
    w[some] = rng.integers(1, wmax + 1, int(some.sum()))
    return cm.Graph(g.xadj, g.adjncy, w, g.vwgt)


GRAPHS = {
    "four": _four,
    "grid": lambda: _changed(cm.gen_grid2d(70, 60), 0.02, 3, 1),
    "rgg": lambda: _changed(cm.gen_rgg(5000, 40.0, seed=2), 0.2, 5, 2),
    "rmat": lambda: _changed(cm.gen_rmat(12, 16, seed=3, wmax=5), 0.01, 5, 3),
    "rmat 16": lambda: _changed(cm.gen_rmat(16, 24, seed=3, wmax=5), 0.01, 5, 3),
}


def _rounds(g, cap, mode):
    """The oracle's matching; one-way pointers can remain, so its rounds are bounded."""
    a = O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt)
    want = O.match_rounds(a, cap, mode, 200)[0]
    assert np.array_equal(want, O.match_rounds(a, cap, mode, 199)[0])
    assert g.nvtxs > 4 or list(want) == [1, 0, 2, 3]
    return want


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_match(ctx, name, mode):
    g = GRAPHS[name]()
    m, _ = ctx.match(g.to_device(), 64, mode)
    assert np.array_equal(m.cpu().numpy(), _rounds(g, 64, mode))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", ["four", "grid", "rgg"])
def test_whole_levels(ctx, name, mode):
    g = GRAPHS[name]()
    h = ctx.coarsen(g.to_device(), 1, mode, maxvwgt=64, max_levels=1)
    assert np.array_equal(h.copy_level(0)[2], _rounds(g, 64, mode))
    h.close()
