"""A 3D graph with more nodes than a launch grid's second dimension has
blocks: single precision runs it as double does."""
import ctypes

import numpy as np
import pytest

from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


def _flat(dt, leaves, its):
    """u and pt of the first leaf and u of all, of a root over `leaves` leaves."""
    from asetsmatlabmaxflow_gb300 import native as N

    D, m, n = (3, 2, 2), leaves + 1, 12
    g = np.random.default_rng(3)
    costs = g.random((leaves, n)).astype(dt)
    out = {k: np.zeros((m, n), dt) for k in ("u", "pt", "pn", "div", "g")}
    flows = [np.zeros((m, f), dt) for f in (8, 6, 6)]
    ptrs = lambda a, lo=0: (ctypes.c_void_p * m)(*([None] * lo + [r.ctypes.data for r in a]))  # noqa: E731
    nchild = np.zeros(m, np.int32)
    nchild[0] = leaves
    kids = np.arange(1, m, dtype=np.int32)
    alpha = np.full(m, 0.2)
    N.check(N.lib().asets_dag_run(
        N.Context.default().handle, np.dtype(dt).itemsize, 3, *D, m, nchild.ctypes.data, kids.ctypes.data,
        ptrs(costs, 1), (ctypes.c_void_p * m)(), alpha.ctypes.data, None, None, None, its, 0.1, 0.25,
        *(ptrs(out[k]) for k in ("u", "pt", "pn", "div", "g")), *(ptrs(f) for f in flows)))
    return out


def test_more_nodes_than_grid_rows():
    require_gpu()
    leaves, its = 65600, 2
    a, b = _flat(np.float32, leaves, its), _flat(np.float64, leaves, its)
    # the root's flow is a sum of `leaves` terms in float, a rounding of at
    # most half an ulp of the running sum each, and twice that in two iterations
    tol = 2 * its * leaves * 2.0 ** -24
    for k in ("u", "pt", "div"):
        size = max(1.0, np.abs(b[k]).max())
        assert np.abs(a[k].astype(np.float64) - b[k]).max() <= tol * size, k
