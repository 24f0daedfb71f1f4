"""Small graphs coarsened by one kernel against the separate kernels (which the
stage timers select), level for level and bit for bit: every family, both tie
orders, level limits, levels that hardly shrink (the allocation runs out), rows
too long for the kernel, and an adjacency that is not symmetric."""
import numpy as np
import pytest

import cumetis_gb300 as cm

pytestmark = pytest.mark.gpu


def _weighted(g, vmax, wmax, seed):
    rng = np.random.default_rng(seed)
    row = np.repeat(np.arange(g.nvtxs), np.diff(g.xadj)).astype(np.int64)
    lo, hi = np.minimum(row, g.adjncy), np.maximum(row, g.adjncy)
    w = 1 + (lo * 1000003 + hi * 7919 + seed) % wmax
    return cm.Graph(g.xadj, g.adjncy, w, rng.integers(1, vmax + 1, g.nvtxs))


def _star_of_paths(arms, length):
    """A hub joined to the ends of `arms` paths."""
    n = 1 + arms * length
    e = [(0, 1 + i * length) for i in range(arms)]
    e += [(1 + i * length + j, 2 + i * length + j) for i in range(arms) for j in range(length - 1)]
    e = np.array(e + [(b, a) for a, b in e])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    return cm.Graph(np.r_[0, np.cumsum(np.bincount(e[:, 0], minlength=n))], e[:, 1])


def _one_way(g, seed):
    keep = np.random.default_rng(seed).random(g.nedges) >= 0.02
    row = np.repeat(np.arange(g.nvtxs), np.diff(g.xadj))
    return cm.Graph(np.r_[0, np.cumsum(np.bincount(row[keep], minlength=g.nvtxs))], g.adjncy[keep], g.adjwgt[keep],
                    g.vwgt)


GRAPHS = {
    "one vertex": lambda: cm.Graph([0, 0], [], [], [3]),
    "one edge": lambda: cm.Graph([0, 1, 2], [1, 0]),
    "no edges": lambda: cm.Graph(np.zeros(700, np.int32), []),
    "path": lambda: cm.gen_grid2d(1500, 1),
    "tri": lambda: cm.gen_tri_grid(69, 69),
    "grid2d": lambda: cm.gen_grid2d(301, 207),
    "grid3d weighted": lambda: _weighted(cm.gen_grid3d(31, 28, 30), 5, 100, 1),
    "rgg": lambda: cm.gen_rgg(40000, 8.0, seed=2),
    "rgg dense": lambda: _weighted(cm.gen_rgg(6000, 40.0, seed=3), 1, 3, 2),      # rows of 65 to 256
    "rgg denser": lambda: cm.gen_rgg(3000, 120.0, seed=4),                         # expanded rows above 256
    "star 300": lambda: _star_of_paths(300, 9),                                    # a row above 256
    "star 200": lambda: _star_of_paths(200, 9),
    "rmat": lambda: cm.gen_rmat(9, 4, seed=5),
    "one way": lambda: _one_way(cm.gen_grid2d(90, 80), 6),
}


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_levels_equal_the_separate_kernels(ctx, name, mode):
    g = GRAPHS[name]()
    for thr, kw in ((max(1, g.nvtxs // 40), {}), (1, {"shrink": 1.0}), (1, {"max_levels": 2, "maxvwgt": 9})):
        hs = []
        for separate in (False, True):
            ctx.set_stage_timing(separate)
            hs.append(ctx.coarsen(g if separate else g.to_device(), thr, mode, **kw))
        ctx.set_stage_timing(False)
        a, b = hs
        assert a.sizes() == b.sizes(), (name, thr)
        for l in range(len(a)):
            x, y = a.copy_level(l), b.copy_level(l)
            for f in ("xadj", "adjncy", "adjwgt", "vwgt"):
                assert np.array_equal(getattr(x[0], f), getattr(y[0], f)), (name, thr, l, f)
            if x[1] is not None:
                assert np.array_equal(x[1], y[1]) and np.array_equal(x[2], y[2]), (name, thr, l)
        a.close()
        b.close()
