"""Small graphs on the device, whose weight limit and longest row the coarsening kernel
finds itself, against the same graphs from the host: rows at the edge of what it
takes, weights whose sum leaves 32 bits, limits given by the caller."""
import numpy as np
import pytest

import cumetis_gb300 as cm

pytestmark = pytest.mark.gpu


def _star(arms, length, vwgt):
    """A hub joined to the ends of `arms` paths."""
    n = 1 + arms * length
    e = [(0, 1 + i * length) for i in range(arms)]
    e += [(1 + i * length + j, 2 + i * length + j) for i in range(arms) for j in range(length - 1)]
    e = np.array(e + [(b, a) for a, b in e])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    return cm.Graph(np.r_[0, np.cumsum(np.bincount(e[:, 0], minlength=n))], e[:, 1], None, np.full(n, vwgt, np.int32))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("vwgt", [1, 2**22])
@pytest.mark.parametrize("arms", [2, 255, 256, 257, 513])
def test_device_input_as_host_input(ctx, arms, vwgt, mode):
    g = _star(arms, 7, vwgt)
    for thr, kw in ((1, {}), (50, {}), (20, {"maxvwgt": 3 * vwgt})):
        a, b = ctx.coarsen(g.to_device(), thr, mode, **kw), ctx.coarsen(g, thr, mode, **kw)
        assert a.sizes() == b.sizes()
        for l in range(len(a)):
            x, y = a.copy_level(l)[0], b.copy_level(l)[0]
            for f in ("xadj", "adjncy", "adjwgt", "vwgt"):
                assert np.array_equal(getattr(x, f), getattr(y, f)), (thr, l, f)
        a.close()
        b.close()
