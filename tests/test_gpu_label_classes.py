"""Default forms of multi-label 2D solves by size and shape class, where the
slower of the two kinds is a tenth or more behind: 32 launches of two passes or
16 of one (a run of 16 iterations), 1 of the whole solve."""
import numpy as np
import pytest

from tests.gpu_helpers import bits, require_gpu
from tests.test_gpu_fused_labels import TWO_PASS, _inputs, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,dims,L,exact,launches", [
    ("ishikawa", (144, 2292), 8, False, 32), ("ishikawa", (2048, 2050), 2, False, 16), ("potts", (300, 2000), 7, False, 16),
    ("potts", (420, 2510), 7, True, 16), ("ishikawa", (400, 1700), 8, False, 16), ("potts", (585, 3504), 3, True, 16),
    ("potts", (442, 339), 5, True, 16), ("ishikawa", (1006, 457), 2, True, 16)])
def test_class_and_result(model, dims, L, exact, launches):
    require_gpu()
    ct, alpha = _inputs(model, dims, L, 3)
    g = _solve(model, dims, L, ct, alpha, 16, 0.0, exact, 0)
    assert g["launches"] == launches
    if exact:
        t = _solve(model, dims, L, ct, alpha, 16, 0.0, True, TWO_PASS)
        for k in ("u", "pt", "bx", "by"):
            np.testing.assert_array_equal(bits(g[k]), bits(t[k]), err_msg=k)
