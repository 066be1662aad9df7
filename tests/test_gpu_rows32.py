"""The labelled 3D kernel's 32-row tiles (one row a lane; tile_config 5 to 7)
at the edges of their 16, 12 and 10 columns: EXACT bits of the oracle, and the
default's for volumes of up to 32 rows."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_helpers import bits, require_gpu
from tests.test_gpu_carry3d import STEPS, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(32, 16, 9), (33, 17, 5), (31, 12, 1), (1, 10, 7), (30, 11, 2), (65, 21, 6)])
@pytest.mark.parametrize("model,L", [("potts", 3), ("ishikawa", 5)])
def test_one_row_a_lane(model, L, dims):
    from asetsmatlabmaxflow_gb300 import native as N

    require_gpu()
    ct, al, _ = _inputs(model, dims, L, 17)
    ref = O.solve(model, dims, ct, al, nlab=L, max_it=9, err_bound=0.0, cc=0.3, steps=STEPS)
    s = N.Solver(N.Context.default(), model, dims, L)
    s.set_inputs(ct, al)
    for tc in (0, 5, 6, 7):
        s.run(9, 0.0, 0.3, STEPS, exact=True, tile_config=tc)
        assert np.array_equal(bits(s.get_u()), bits(ref["u"].ravel(order="F")))
        # nine iterations of at most a few ulp of O(1) each
        s.run(9, 0.0, 0.3, STEPS, tile_config=tc)
        assert float(np.max(np.abs(s.get_u() - ref["u"].ravel(order="F")))) <= 1e-5
    s.close()
