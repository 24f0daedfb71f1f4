"""Bucket-sorted coarse rows: ids spread evenly, in clusters, all equal, and in
orders that leave the bucket bounds useless, against the oracle.  Integer work:
every comparison is bit-exact."""
import numpy as np
import pytest

import cumetis_gb300 as cm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _row_ids(kind, L, n, rng):
    if kind == "spread":
        return np.sort(rng.choice(n, L, replace=False))
    if kind == "clusters":  # runs of consecutive ids far apart
        runs = max(1, L // 25)
        base = np.sort(rng.choice(n - 30, runs, replace=False))
        return np.unique(np.concatenate([b + np.arange(-(-L // runs)) for b in base]))[:L]
    if kind == "equal":  # parallel entries
        return np.full(L, rng.integers(n))
    if kind == "few":
        return np.sort(rng.choice(rng.choice(n, 3, replace=False), L))
    if kind == "skewed":  # most ids low
        return np.sort((n * rng.random(L) ** 12).astype(np.int64))
    ids = rng.choice(n, L, replace=False)  # "inner": the ends of the row are its middle ids
    ids.sort()
    m = L // 2
    return np.r_[ids[m:m + 1], rng.permutation(np.delete(ids, [m, min(m + 1, L - 1)])), ids[min(m + 1, L - 1):m + 2]][:L]


@pytest.mark.parametrize("kind", ["spread", "clusters", "equal", "few", "skewed", "inner"])
@pytest.mark.parametrize("lens", [(1, 2, 3, 5, 16, 31, 32, 33, 48), (33, 47, 64, 95, 96, 100, 128, 191, 250),
                                  (256, 300, 383, 511, 700, 1023, 1400, 2047), (2500, 4000, 6000, 8191)])
def test_rows_of_every_shape(ctx, kind, lens):
    """Every row twice, the copies paired, so that an expanded row has up to
    2 L entries with every id twice; the leaves are paired with a neighbour or
    left alone.  Weights include 2^30: merged weights wrap."""
    import torch
    rng = np.random.default_rng(len(kind) * 100 + lens[0])
    nh, n = 2 * len(lens), 40000
    src, dst = [], []
    for i, L in enumerate(lens):
        for r in (2 * i, 2 * i + 1):
            ids = _row_ids(kind, L, n - nh, rng) + nh
            src.append(np.full(len(ids), r))
            dst.append(ids)
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.choice(np.array([1, 5, 1 << 30], np.int64), len(src))
    order = np.argsort(dst, kind="stable")  # the leaves' rows: reverse entries
    s2, d2, w2 = np.r_[src, dst[order]], np.r_[dst, src[order]], np.r_[w, w[order]]
    xadj = np.r_[0, np.cumsum(np.bincount(s2, minlength=n))]
    g = O.CSR(xadj, d2, w2.astype(np.int32), np.ones(n))
    match = np.arange(n, dtype=np.int32)
    pair = np.arange(0, n, 2)
    pair = pair[(pair < nh) | (rng.random(len(pair)) < 0.5)]
    match[pair], match[pair + 1] = pair + 1, pair
    want, wcmap = O.contract(g, match)
    cg, cmap = ctx.contract(cm.Graph(g.xadj, g.adjncy, g.adjwgt, g.vwgt).to_device(),
                            torch.from_numpy(match).cuda())
    h = cg.to_host()
    assert np.array_equal(cmap.cpu().numpy(), wcmap)
    for f in ("xadj", "adjncy", "adjwgt", "vwgt"):
        assert np.array_equal(getattr(h, f), getattr(want, f)), f
