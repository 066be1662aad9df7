"""The Matlab-semantics solvers on capacities and costs that are not ordinary
numbers: values and NaN places of the numpy restatement."""
import numpy as np
import pytest

from oracle import mtwin as M
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu

VALUES = {"alpha": (np.nan, np.inf, 0.0, -1.0, 1e-300, 1e300), "costs": (np.nan, np.inf, -np.inf, 1e300, -0.0)}


# the last: large enough for the one-pass form in single precision
@pytest.mark.parametrize("shape,its", [((40, 30), 6), (((21, 20, 9)), 6), ((64, 60, 53), 2)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("what", sorted(VALUES))
def test_special_values(what, dtype, shape, its):
    from asetsmatlabmaxflow_gb300 import matlab

    require_gpu()
    g = np.random.default_rng(8)
    cs, ct = (g.random(shape).astype(dtype) for _ in range(2))
    al = (0.02 + 0.2 * g.random(shape)).astype(dtype)
    with np.errstate(all="ignore"):
        for v in VALUES[what]:
            for a in ((al,) if what == "alpha" else (cs, ct)):
                a[tuple(g.integers(1, n - 1) for n in shape)] = dtype(v)
        steps = 0.11 if len(shape) == 3 else 0.16
        ref = M.binary(cs, ct, al, its, 1e-30, 0.3, steps)
    fn = matlab.asetsBinaryMF3D if len(shape) == 3 else matlab.asetsBinaryMF2D
    got = fn(cs, ct, al, [*shape, its, 1e-30, 0.3, steps])
    assert np.isnan(ref[0]).any() and got[2] == ref[2]
    assert np.array_equal(got[0], ref[0], equal_nan=True)

