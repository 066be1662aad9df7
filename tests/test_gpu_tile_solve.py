"""Whole-solve launches whose blocks keep their tile on chip or take several,
and the block sums of erriter: EXACT state bit for bit against the two-pass
form or the oracle, and infinite and NaN sums as the oracle has them."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_helpers import bits, require_gpu
from tests.test_gpu_fused_labels import TWO_PASS, _inputs, _solve
from tests.test_gpu_tile2d import SWEEP, TILE_EXACT

pytestmark = pytest.mark.gpu

WHOLE = 5  # tile_config of the multi-label whole-solve form


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


# more tiles than blocks (one block an SM at eight labels); one tile; tiles cut
# by one row and column; a single row
@pytest.mark.parametrize("model,dims,L", [
    ("potts", (400, 380), 8), ("ishikawa", (300, 401), 9), ("potts", (16, 16), 3), ("ishikawa", (17, 33), 6),
    ("potts", (1, 40), 5), ("ishikawa", (49, 1), 4)])
def test_labelled_whole_solve(model, dims, L):
    ct, alpha = _inputs(model, dims, L, 5)
    g = _solve(model, dims, L, ct, alpha, 9, 0.0, True, WHOLE)
    t = _solve(model, dims, L, ct, alpha, 9, 0.0, True, TWO_PASS)
    assert g["launches"] == 1
    for k in ("u", "pt", "bx", "by"):
        np.testing.assert_array_equal(bits(g[k]), bits(t[k]), err_msg=k)
    # float shares of at most 13 terms each, summed to well below a float's ulp
    np.testing.assert_allclose(g["cvg"], t["cvg"], rtol=26 * 2.0 ** -24, atol=1e-30)


@pytest.mark.parametrize("tc", (SWEEP,) + TILE_EXACT)
@pytest.mark.parametrize("value", [-np.inf, np.nan, -3e38])
def test_sums_that_are_not_finite(tc, value):
    from asetsmatlabmaxflow_gb300 import native as N

    dims = (40, 33)
    g = np.random.default_rng(2)
    cs, ct, al = (np.asfortranarray(g.random(dims).astype(np.float32)) for _ in range(3))
    ct[7, 5] = value
    with np.errstate(all="ignore"):
        ref = O.solve("binary", dims, ct, al, cs=cs, max_it=3, err_bound=0.0, cc=0.3, steps=0.16)
    s = N.Solver(N.Context.default(), "binary", dims)
    s.set_inputs(ct, al, cs)
    s.run(3, 0.0, 0.3, 0.16, exact=True, tile_config=tc)
    cvg = s.get_cvg()
    s.close()
    np.testing.assert_array_equal(np.isnan(cvg), np.isnan(ref["cvg"]))
    np.testing.assert_array_equal(np.isinf(cvg), np.isinf(ref["cvg"]))
