"""Host graphs whose arrays start between two words, and levels read into such arrays."""
import numpy as np
import pytest

import cumetis_gb300 as cm

pytestmark = pytest.mark.gpu


def _odd(a, by):
    raw = np.zeros(4 * len(a) + 8, np.uint8)
    raw[by:by + 4 * len(a)] = np.ascontiguousarray(a, np.int32).view(np.uint8)
    return np.frombuffer(raw, np.int32, len(a), by)


@pytest.mark.parametrize("by", [1, 2, 3])
def test_arrays_off_a_word(ctx, by):
    g = cm.gen_grid2d(37, 41)
    p = cm.Graph(*(_odd(a, by) for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt)))
    hs = [ctx.coarsen(p, 1, max_levels=1), ctx.coarsen_batch([p], 1, max_levels=1)[0]]
    for h in hs:
        out = [_odd(np.zeros(len(a)), by) for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt)]
        h.read_level(0, *[a.ctypes.data for a in out])
        for a, f in zip(out, ("xadj", "adjncy", "adjwgt", "vwgt")):
            assert np.array_equal(a, getattr(g, f)), f
        h.close()
