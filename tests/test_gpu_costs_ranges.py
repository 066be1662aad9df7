"""Contrast weights and normalised costs of images whose range is tiny, huge
or beyond the float range: the quotients' own values."""
import numpy as np
import pytest

from oracle import costs as C
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(0.0, 1.0), (-3e38, 3e38), (0.0, 3e38), (1e38, 3e38), (0.0, 1e-38), (-1e30, 1e31),
                                   (0.0, np.inf), (-np.inf, 1.0)])
def test_contrast_of_any_range(lo, hi):
    from asetsmatlabmaxflow_gb300 import costs

    require_gpu()
    g = np.random.default_rng(1)
    img = np.asfortranarray(g.random((12, 9, 5)).astype(np.float32))
    a, b = (max(min(v, 3e38), -3e38) for v in (lo, hi))
    with np.errstate(all="ignore"):
        img = np.asfortranarray((np.float32(a) * (1 - img) + np.float32(b) * img).astype(np.float32))
        img[3, 4, 2], img[8, 1, 1] = lo, hi
        ref = C.alpha_contrast(img, 0.05, 0.3, 10.0)
    got = costs.alpha_contrast(img, 0.05, 0.3, 10.0)
    # as for ordinary images: four half-ulps of the gradient, times c b = 3
    np.testing.assert_allclose(got, ref, rtol=1e-6, atol=1e-6)


def test_quotients_below_the_normal_range():
    """Values of 2^-95 and less over a range of 2^40: IEEE quotients."""
    from asetsmatlabmaxflow_gb300 import costs

    require_gpu()
    g = np.random.default_rng(2)
    img = np.ldexp(g.random(4000).astype(np.float32), -95 - g.integers(0, 20, 4000)).astype(np.float32)
    img[0], img[1] = 0.0, 2.0 ** 40 * 1.3
    got = costs.l1(img.reshape(-1, 1), [0.0])
    assert np.array_equal(got.ravel().view(np.uint32), C.cost_l1(img, [0.0]).ravel().view(np.uint32))
