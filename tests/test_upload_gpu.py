"""Host graphs whose arrays start off a 16-byte boundary, end inside a 64 KB
piece, and are more than one upload launch takes, arrive unchanged."""
import numpy as np
import pytest

import cumetis_gb300 as cm

pytestmark = pytest.mark.gpu


def _shifted(a, by):
    buf = np.zeros(len(a) + by, np.int32)
    buf[by:] = a
    return buf[by:]


@pytest.mark.parametrize("by", [0, 1, 3])
def test_host_arrays_arrive(ctx, by):
    sizes = [1, 2, 7, 4095, 4096, 4097, 16383, 16384, 16385, 40001] * 4  # 160 arrays
    gs = []
    for i, n in enumerate(sizes):
        g = cm.gen_grid2d(n, 1)
        w = (np.arange(g.nedges) * 7919 + i) % 1000003
        gs.append(cm.Graph(*(_shifted(np.asarray(a, np.int32), by) for a in
                             (g.xadj, g.adjncy, w, 1 + np.arange(n) % 5))))
    for hs in (ctx.coarsen_batch(gs, 1, max_levels=1), [ctx.coarsen(g, 1, max_levels=1) for g in gs[:12]]):
        for g, h in zip(gs, hs):
            got, _, _ = h.copy_level(0)
            for f in ("xadj", "adjncy", "adjwgt", "vwgt"):
                assert np.array_equal(getattr(got, f), getattr(g, f)), (g.nvtxs, f)
            h.close()
