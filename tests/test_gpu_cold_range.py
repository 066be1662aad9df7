"""The cold start's joint state of pt and u at the edges of its range: small
costs, whose u is small for many iterations, step parameters on both sides of
the rule, costs around its limit."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu

DIMS = (40, 22, 10)


def _inputs(scale, seed=3):
    g = np.random.default_rng(seed)
    return [np.asfortranarray((scale * (0.05 + g.random(DIMS))).astype(np.float32)) for _ in range(3)]


def _solve(cs, ct, al, cc, its):
    from asetsmatlabmaxflow_gb300 import native as N

    require_gpu()
    s = N.Solver(N.Context.default(), "binary", DIMS)
    s.set_inputs(ct, al, cs)
    s.run(its, 0.0, cc, 0.11)
    u = s.get_u()
    s.close()
    return u, O.solve("binary", DIMS, ct, al, cs=cs, max_it=its, err_bound=0.0, cc=cc,
                      steps=0.11)["u"].ravel(order="F")


@pytest.mark.parametrize("scale", [1e-12, 1e-15])
def test_small_costs_move_u(scale):
    """u starts at 0 where Cs < Ct and moves, beside a block where it is 1, by
    cc times divergences of the size of the capacities (there the flows are
    full): kept to some sixty roundings of such terms an iteration."""
    cs, ct, al = _inputs(scale)
    cs[:] = np.float32(0.9) * ct
    cs[10:30, 5:15, 3:7] *= np.float32(1.3)
    its = 4
    u, ref = _solve(cs, ct, al, 2.0 ** -4, its)
    small = ref < 0.5
    assert (ref[small] > 0).sum() > 100 and ref[small].max() < scale
    assert np.abs(u - ref)[small].max() <= 64 * its * scale * 2.0 ** -24


@pytest.mark.parametrize("cc", [-0.3, 2.0, 700.0, 1e-3])
def test_step_parameters_out_of_the_rule(cc):
    """Whatever cc, fast and reference iterations agree to roundings: at most
    some thirty of terms of the size of max(1, cc, 1/cc) an iteration."""
    cs, ct, al = _inputs(1.0)
    its = 4
    u, ref = _solve(cs, ct, al, cc, its)
    size = max(1.0, abs(cc), 1.0 / abs(cc), float(np.abs(ref).max()))
    assert np.isfinite(ref).all() and np.abs(u - ref).max() <= 30 * its * size * max(1.0, abs(cc)) * 2.0 ** -24


@pytest.mark.parametrize("value", [2.0 ** 33, 2.0 ** 34, 2.0 ** 50])
def test_costs_large_on_both_sides(value):
    """Cells whose two costs are both huge: u there is cc times roundings of
    such values and may be far above 2^14; the others are as ever."""
    cs, ct, al = _inputs(1.0)
    cs[5:9, 3:6, 4] = value
    ct[5:9, 3:6, 4] = value * 1.5
    its = 8
    u, ref = _solve(cs, ct, al, 0.3, its)
    err = np.abs(u - ref).reshape(DIMS, order="F")
    far = np.ones(DIMS, bool)
    far[3:11, 1:8, 2:7] = False
    assert err[far].max() <= 1e-3
    assert err.max() <= 1.0 + 30 * its * value * 2.0 ** -24
