"""The Matlab-semantics solvers on strips: tiles of 4, 8 and 16 rows, whose
widths are 64, 32 and 16 columns in the step and half that in the update, at the
edges of both, and the volumes either side of the one-pass form's 24 rows."""
import numpy as np
import pytest

from tests.gpu_helpers import require_gpu
from tests.test_gpu_matlab_tiles import _check, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(1, 65), (4, 64), (5, 63), (8, 33), (9, 32), (16, 17), (17, 40), (24, 9), (40, 16),
                                   (3, 33, 5), (8, 31, 3), (12, 15, 4), (36, 20, 2)])
@pytest.mark.parametrize("model,L", [("binary", 1), ("potts", 3), ("potts", 7), ("ishikawa", 4)])
def test_strips(model, L, shape, dtype):
    require_gpu()
    _check(*_run(model, shape, L, dtype, 11, its=12), dtype)


@pytest.mark.parametrize("shape", [(23, 100, 90), (24, 100, 90)])
def test_one_pass_rows(shape):
    require_gpu()
    _check(*_run("binary", shape, 1, np.float32, 12, its=4), np.float32)
