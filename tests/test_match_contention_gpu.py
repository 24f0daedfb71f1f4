"""Matchings in which many warps displace one another's vertices at the same
time: every row is longer than a lane's scan, few distinct weights make the
candidates' proposals change while they are looked at, and tight vertex weights
make lists end early.  Bit-exact against the oracle."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("wmax,vmax,cap", [(1, 1, 100), (3, 5, 7), (100, 5, 9)])
@pytest.mark.parametrize("n,degree", [(600, 30.0), (20000, 40.0), (9000, 110.0)])
def test_warps_that_displace_one_another(ctx, n, degree, wmax, vmax, cap, mode):
    g = cm.gen_rgg(n, degree, seed=n + wmax)
    row = np.repeat(np.arange(n, dtype=np.int64), np.diff(g.xadj))
    lo, hi = np.minimum(row, g.adjncy), np.maximum(row, g.adjncy)
    w = 1 + (lo * 1000003 + hi * 7919) % wmax
    v = np.random.default_rng(n).integers(1, vmax + 1, n)
    want = O.match_greedy(O.CSR(g.xadj, g.adjncy, w, v), cap, mode)
    d = cm.Graph(g.xadj, g.adjncy, w, v).to_device()
    for _ in range(5):
        m, _ = ctx.match(d, cap, mode)
        assert np.array_equal(m.cpu().numpy(), want)
