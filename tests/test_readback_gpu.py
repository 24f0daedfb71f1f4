"""Levels read back into host arrays: sizes at the edges of a page, a piece and the
limit between the kernel and the copy calls, off a 16-byte boundary, in pageable and
pinned memory, with nothing written outside the arrays."""
import numpy as np
import pytest
import torch

import cumetis_gb300 as cm

pytestmark = pytest.mark.gpu


def _buffer(n, by, pinned):
    t = torch.full((n + by + 8,), -7, dtype=torch.int32, pin_memory=pinned)
    return t, t.numpy()[by:by + n]


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n", [1, 2, 1023, 1025, 16384, 16385, 40001, 90001, 1398100, 1398102])
def test_read_level(ctx, n, pinned):
    g = cm.gen_grid2d(n, 1)
    g = cm.Graph(np.asarray(g.xadj, np.int32), np.asarray(g.adjncy, np.int32),
                 ((np.arange(g.nedges) * 7919) % 1000003).astype(np.int32), (1 + np.arange(n) % 5).astype(np.int32))
    h = ctx.coarsen(g, 1, max_levels=1)
    want = [np.asarray(a) for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt)]
    for by in (0, 1, 3):
        bufs = [_buffer(len(a), by, pinned) for a in want]
        h.read_level(0, *[b.ctypes.data for _, b in bufs])
        for w, (t, b) in zip(want, bufs):
            assert np.array_equal(w, b)
            assert (t[:by] == -7).all() and (t[by + len(w):] == -7).all()
    got, cmap, match = h.copy_level(0)
    for w, f in zip(want, ("xadj", "adjncy", "adjwgt", "vwgt")):
        assert np.array_equal(w, np.asarray(getattr(got, f)))
    h.close()
