"""The hierarchical solver's passes where they are cut: the 28-row strips and
the column runs of the 2D sweep, the two 3D passes, pixel counts that end
within a 16-byte vector, trees either side of the staged per-pixel pass's 18
nodes, alphas of which no flow is inside, divisors that are a power of two or
not.  Every state array bit for bit against the restatement (oracle/hmf.py)."""
import numpy as np
import pytest

from oracle import hmf as H
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


def _tree(make, img, alphas, leaves):
    dt = img.dtype.type
    lv = [make([], alphas[i % len(alphas)], np.abs(img - dt(i / max(leaves - 1, 1))).astype(img.dtype))
          for i in range(leaves)]
    half = leaves // 2
    return make([make(lv[:half], alphas[0])] + lv[half:], 0)


def _check(shape, dtype, alphas, leaves, its, cc):
    from asetsmatlabmaxflow_gb300.hmf import asetsHMF2D, asetsHMF3D

    img = np.random.default_rng(sum(shape) + leaves).random(shape).astype(dtype)
    alphas = [np.asarray(a, dtype) if np.ndim(a) else a for a in alphas]
    ref = _tree(H.Node, img, alphas, leaves)
    gpu = _tree(asetsHMF2D if len(shape) == 2 else asetsHMF3D, img, alphas, leaves)
    ref.max_full_flow(its, 0.1, cc)
    gpu.MaxFullFlow(its, 0.1, cc)
    bits = lambda a: np.ascontiguousarray(a).view(np.uint64 if dtype == np.float64 else np.uint32)  # noqa: E731
    for r, q in zip(H.preorder(ref), gpu._nodes()):
        for name in ("u", "pt", "div", "g"):
            assert np.array_equal(bits(getattr(q, name)), bits(getattr(r, name))), name
        for k, name in enumerate(("px", "py", "pz")[:len(shape)]):
            assert np.array_equal(bits(getattr(q, name)), bits(r.p[k])), name


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(1, 1), (2, 1), (28, 3), (29, 7), (27, 8), (56, 33), (57, 61), (301, 203),
                                   (33, 9, 5), (1, 6, 7), (5, 1, 3), (31, 17, 13)])
def test_cut_passes(shape, dtype):
    """Small alphas, so that flows are inside and outside of them."""
    _check(shape, dtype, [0.02, 0.05], 4, 30, 0.25 if sum(shape) % 2 else 0.2)


@pytest.mark.parametrize("dtype,leaves", [(np.float32, 16), (np.float32, 17), (np.float64, 16), (np.float64, 17)])
def test_trees_either_side_of_the_staged_limit(dtype, leaves):
    _check((31, 19), dtype, [0.05], leaves, 12, 0.25)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_alpha_extremes(dtype):
    shape = (37, 23)
    g = np.random.default_rng(1)
    a = 0.05 * g.random(shape)
    a[g.random(shape) < 0.2] = 0.0
    a[g.random(shape) < 0.1] = np.inf
    a[g.random(shape) < 0.1] = 1e-30
    _check(shape, dtype, [a], 4, 15, 0.25)
