"""Stars: a warp's vertices that all want the same neighbour.  Bit-exact against the
oracle, with the hub first, last and in the middle, leaves that fill warps or not,
equal and different weights, and leaves joined in pairs, which go on with each other."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("wmax", [1, 4, 1000000])
@pytest.mark.parametrize("leaves", [1, 31, 32, 33, 64, 1023, 30000])
def test_star(ctx, leaves, wmax, mode):
    rng = np.random.default_rng(leaves + wmax)
    for hub in (0, leaves // 2, leaves):
        leaf = np.delete(np.arange(leaves + 1), hub)
        for pairs in (0, leaves // 2):
            a = np.r_[np.full(leaves, hub), leaf[:2 * pairs:2]]
            b = np.r_[leaf, leaf[1:2 * pairs:2]]
            w = np.r_[rng.integers(1, wmax + 1, leaves), np.ones(pairs, np.int64)]
            s, d, x = np.r_[a, b], np.r_[b, a], np.r_[w, w]
            order = np.lexsort((d, s))
            g = cm.Graph(np.r_[0, np.cumsum(np.bincount(s, minlength=leaves + 1))], d[order], x[order])
            want = O.match_greedy(O.CSR(g.xadj, g.adjncy, g.adjwgt, g.vwgt), 100, mode)
            got = ctx.match(g.to_device(), 100, mode)[0].cpu().numpy()
            assert np.array_equal(got, want), (hub, pairs)
