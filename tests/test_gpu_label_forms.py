"""The default form of multi-label 2D solves on either side of its lines: the
EXACT result of whatever form runs is the two-pass form's, and the launch count
tells that the line lies where it is drawn."""
import numpy as np
import pytest

from tests.gpu_helpers import bits, require_gpu
from tests.test_gpu_fused_labels import TWO_PASS, _inputs, _solve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


# launches of a run of 16 iterations (a chunk holds 16): 1 whole solve, 16 one
# pass, 32 two passes
@pytest.mark.parametrize("model,dims,L,exact,launches", [
    ("potts", (512, 512), 2, False, 1), ("potts", (440, 440), 4, False, 32), ("potts", (548, 548), 4, False, 16),
    ("potts", (547, 547), 4, False, 32), ("potts", (700, 660), 2, False, 32), ("potts", (180, 1700), 5, False, 32),
    ("potts", (1700, 180), 5, False, 32), ("potts", (1700, 180), 6, False, 16), ("potts", (440, 440), 5, True, 1),
    ("potts", (440, 440), 6, True, 32), ("potts", (500, 501), 6, True, 16), ("ishikawa", (512, 512), 4, True, 1),
    ("ishikawa", (512, 512), 5, True, 16), ("ishikawa", (640, 480), 9, False, 16)])
def test_form_and_result(model, dims, L, exact, launches):
    ct, alpha = _inputs(model, dims, L, 3)
    g = _solve(model, dims, L, ct, alpha, 16, 0.0, exact, 0)
    assert g["launches"] == launches
    if exact:
        t = _solve(model, dims, L, ct, alpha, 16, 0.0, True, TWO_PASS)
        for k in ("u", "pt", "bx", "by"):
            np.testing.assert_array_equal(bits(g[k]), bits(t[k]), err_msg=k)
