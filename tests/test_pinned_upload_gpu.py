"""Pinned host graphs around the size from which the copy engines take an array, whole
and off a 16-byte boundary, arrive unchanged beside arrays that the kernel takes."""
import numpy as np
import pytest
import torch

import cumetis_gb300 as cm

pytestmark = pytest.mark.gpu


def _pinned(a, by):
    t = torch.zeros(len(a) + by, dtype=torch.int32, pin_memory=True)
    b = t.numpy()[by:]
    b[:] = a
    return b


@pytest.mark.parametrize("by", [0, 1])
@pytest.mark.parametrize("n", [1000, 131072, 131073, 131074, 262143, 262144])
def test_pinned_arrays_arrive(ctx, n, by):
    g = cm.gen_grid2d(n, 1)
    w = (np.arange(g.nedges) * 7919) % 1000003
    p = cm.Graph(*(_pinned(np.asarray(a, np.int32), by) for a in (g.xadj, g.adjncy, w, 1 + np.arange(n) % 5)))
    assert p.adjncy.ctypes.data % 16 == 4 * by
    for h in (ctx.coarsen(p, 1, max_levels=1), ctx.coarsen_batch([p], 1, max_levels=1)[0]):
        got, _, _ = h.copy_level(0)
        for f in ("xadj", "adjncy", "adjwgt", "vwgt"):
            assert np.array_equal(getattr(got, f), getattr(p, f)), f
        h.close()
