"""Contrast weights of images whose columns share a warp: rows of 1 to 16
lanes of one and of four rows, column counts either side of a block's."""
import numpy as np
import pytest

from oracle import costs as C
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 257, 2), (2, 129, 3), (3, 81, 1), (5, 47, 2), (7, 33, 17), (11, 17, 2), (15, 16, 3),
                                   (16, 65, 2), (17, 9, 2), (4, 255, 2), (8, 129, 3), (20, 48, 2), (20, 49, 2), (64, 17, 2),
                                   (68, 9, 2)])
def test_short_columns(shape):
    from asetsmatlabmaxflow_gb300 import costs

    require_gpu()
    img = np.asfortranarray((np.random.default_rng(4).random(shape) * 300.0 - 20.0).astype(np.float32))
    got = costs.alpha_contrast(img, 0.05, 0.3, 10.0, labels=2)
    ref = C.alpha_contrast(img, 0.05, 0.3, 10.0)
    for l in range(2):  # four half-ulps of the gradient, times c b = 3
        np.testing.assert_allclose(got[..., l], ref, rtol=1e-6, atol=1e-6)
