"""The matching's work split: rows at the edges of the lane, chunk and
multi-chunk scans, and adjacencies that are not symmetric, against the oracle.
Integer work: every comparison is bit-exact."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _match(ctx, g, maxvwgt, mode):
    m, _ = ctx.match(cm.Graph(g.xadj, g.adjncy, g.adjwgt, g.vwgt).to_device(), maxvwgt, mode)
    return m.cpu().numpy()


def _hubs(degrees, copies, wmax, seed):
    """`copies` hubs of every given degree over shared leaves, so that hubs
    displace one another and use their lists up; weights in [1, wmax]."""
    rng = np.random.default_rng(seed)
    nh, nleaf = len(degrees) * copies, 2 * max(degrees)
    src, dst = [], []
    for i in range(nh):
        d = degrees[i % len(degrees)]
        src.append(np.full(d, i))
        dst.append(nh + rng.choice(nleaf, d, replace=False))
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.integers(1, wmax + 1, len(src))
    s2, d2, w2 = np.r_[src, dst], np.r_[dst, src], np.r_[w, w]
    order = np.lexsort((d2, s2))
    xadj = np.r_[0, np.cumsum(np.bincount(s2, minlength=nh + nleaf))]
    return O.CSR(xadj, d2[order], w2[order], 1 + np.arange(nh + nleaf) % 2)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("wmax", [1, 3, 1000])
def test_rows_at_the_scan_boundaries(ctx, mode, wmax):
    """Degrees around a lane's 16 entries, a chunk's 256 and several chunks,
    all weights equal, many ties, few ties; vertex weights that all fit the
    cap, and a cap of 2 that lets only light pairs match."""
    g = _hubs([1, 4, 5, 15, 16, 17, 31, 33, 255, 256, 257, 511, 513, 1300], 6, wmax, seed=wmax)
    for cap in (1000, 4, 3):
        assert np.array_equal(_match(ctx, g, cap, mode), O.match_greedy(g, cap, mode)), (mode, wmax, cap)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("scale,ef", [(9, 4), (12, 16), (16, 24)])
def test_asymmetric_adjacency(ctx, mode, scale, ef):
    """Some entries without their reverse (the largest size takes the
    many-block handshakes): the matching of mutual proposals."""
    g = cm.gen_rmat(scale, ef, seed=scale, wmax=5)
    rng = np.random.default_rng(scale)
    keep = rng.random(g.nedges) >= 0.03
    row = np.repeat(np.arange(g.nvtxs), np.diff(g.xadj))
    xadj = np.r_[0, np.cumsum(np.bincount(row[keep], minlength=g.nvtxs))]
    a = O.CSR(xadj, g.adjncy[keep], g.adjwgt[keep], g.vwgt)
    # one-way pointers remain at the end, so the rounds are bounded (at most 25 are needed)
    want, _ = O.match_rounds(a, 64, mode, 60)
    assert np.array_equal(want, O.match_rounds(a, 64, mode, 59)[0])
    assert np.array_equal(_match(ctx, a, 64, mode), want)
