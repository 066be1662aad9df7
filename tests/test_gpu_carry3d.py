"""3D iteration kernel with the carried gradient source: every tile width at
the edges of its tiles, the flows formed on request, and the cold start's
joint state of pt and u beside the general one."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_helpers import bits, require_gpu

pytestmark = pytest.mark.gpu
STEPS = 0.11


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


def _inputs(model, dims, L, seed):
    g = np.random.default_rng(seed)
    lab = (L,) if model != "binary" else ()
    la = (L - 1,) if model == "ishikawa" else lab
    ct = np.asfortranarray(g.random(dims + lab).astype(np.float32))
    al = np.asfortranarray((0.05 + 0.3 * g.random(dims + la)).astype(np.float32))
    cs = np.asfortranarray(g.random(dims).astype(np.float32)) if model == "binary" else None
    return ct, al, cs


# rows either side of the 64-row tile and its pairs, columns either side of
# the 12, 13, 14 and 16 column tiles, one to a few planes, pitch 4-row padding
SHAPES = [(64, 14, 9), (65, 15, 5), (63, 13, 1), (129, 17, 2), (128, 16, 12), (1, 33, 7), (66, 1, 3),
          (3, 29, 40), (33, 25, 11)]


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("model,L", [("binary", 1), ("potts", 3), ("potts", 7), ("ishikawa", 4)])
def test_every_width_matches_the_oracle(model, L, dims):
    from asetsmatlabmaxflow_gb300 import native as N

    ct, al, cs = _inputs(model, dims, L, 11)
    ref = O.solve(model, dims, ct, al, cs=cs, nlab=L, max_it=9, err_bound=0.0, cc=0.3, steps=STEPS)
    s = N.Solver(N.Context.default(), model, dims, L)
    s.set_inputs(ct, al, cs)
    for tc in range(0, 5):
        s.run(9, 0.0, 0.3, STEPS, exact=True, tile_config=tc)
        assert np.array_equal(bits(s.get_u()), bits(ref["u"].ravel(order="F")))
        # nine iterations of at most a few ulp of O(1) each
        s.run(9, 0.0, 0.3, STEPS, tile_config=tc)
        assert float(np.max(np.abs(s.get_u() - ref["u"].ravel(order="F")))) <= 1e-5
    s.close()


@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("model,L", [("binary", 1), ("potts", 3), ("potts", 7)])
def test_flows_belong_to_the_run_that_left_them(model, L, exact):
    """ps and pt read after the next inputs are set are the last run's; a
    second read, u first or last, and maxIt = 0 give the same state."""
    from asetsmatlabmaxflow_gb300 import native as N

    dims = (37, 18, 6)
    ct, al, cs = _inputs(model, dims, L, 3)
    a = N.Solver(N.Context.default(), model, dims, L)
    a.set_inputs(ct, al, cs)
    a.run(8, 0.0, 0.3, STEPS, exact=exact)
    u, (ps, pt) = a.get_u().copy(), [f.copy() for f in a.get_flows()]
    a.run(8, 0.0, 0.3, STEPS, exact=exact)
    ct2, al2, cs2 = _inputs(model, dims, L, 4)
    a.set_inputs(ct2, al2, cs2)
    ps1, pt1 = a.get_flows()
    assert np.array_equal(bits(ps1), bits(ps)) and np.array_equal(bits(pt1), bits(pt))
    assert np.array_equal(bits(a.get_u()), bits(u))
    a.run(0, 0.0, 0.3, STEPS, exact=exact)
    ref = O.solve(model, dims, ct2, al2, cs=cs2, nlab=L, max_it=0, err_bound=0.0, cc=0.3, steps=STEPS)
    assert np.array_equal(bits(a.get_u()), bits(ref["u"].ravel(order="F")))
    ps0, _ = a.get_flows()
    m = np.minimum(ct2, cs2) if model == "binary" else ct2.min(axis=-1)
    assert np.array_equal(bits(ps0), bits(m.ravel(order="F")))
    a.close()


def test_cold_state_equals_the_general_form():
    """A fast cold start keeps pt and u in one array; the same start given
    explicitly keeps both.  Both stay within the rounding of 30 iterations."""
    from asetsmatlabmaxflow_gb300 import native as N

    dims = (70, 31, 20)
    ct, al, cs = _inputs("binary", dims, 1, 5)
    u0 = (cs - ct >= 0).astype(np.float32)
    m = np.minimum(cs, ct)
    a = N.Solver(N.Context.default(), "binary", dims)
    a.set_inputs(ct, al, cs)
    a.run(30, 0.0, 0.3, STEPS)
    ua, (psa, pta) = a.get_u().copy(), [f.copy() for f in a.get_flows()]
    fa = [f.copy() for f in a.get_spatial_flows()]
    a.set_initial(u0, m, m)
    a.run(30, 0.0, 0.3, STEPS)
    psb, ptb = a.get_flows()
    for x, y in [(ua, a.get_u()), (psa, psb), (pta, ptb)] + list(zip(fa, a.get_spatial_flows())):
        # 30 iterations, a few half-ulps of values up to 1/cc + 1 < 8 each
        assert float(np.max(np.abs(x - y))) <= 30 * 4 * 8 * 2.0 ** -24
    # flows given without u, ps, pt: the cold multipliers on those flows
    a.set_initial(None, None, None)
    a.set_initial_flows(*fa)
    a.run(5, 0.0, 0.3, STEPS)
    uc = a.get_u().copy()
    a.set_initial(u0, m, m)
    a.set_initial_flows(*fa)
    a.run(5, 0.0, 0.3, STEPS)
    assert np.array_equal(bits(uc), bits(a.get_u()))
    a.close()


@pytest.mark.parametrize("value", [1e10, 1e30, np.inf])
def test_hard_constraints_as_large_costs(value):
    """Capacities that force a cell to one side, up to infinity (beyond 2^60
    the general form runs): finite results that match the oracle."""
    from asetsmatlabmaxflow_gb300 import native as N

    dims = (40, 22, 10)
    ct, al, cs = _inputs("binary", dims, 1, 6)
    ct[3:7, 4:9, 2] = value
    cs[20:24, 4:9, 5] = value
    ref = O.solve("binary", dims, ct, al, cs=cs, max_it=25, err_bound=0.0, cc=0.3, steps=STEPS)
    assert np.all(np.isfinite(ref["u"]))
    s = N.Solver(N.Context.default(), "binary", dims)
    s.set_inputs(ct, al, cs)
    s.run(25, 0.0, 0.3, STEPS)
    assert float(np.max(np.abs(s.get_u() - ref["u"].ravel(order="F")))) <= 1e-3
    s.run(25, 0.0, 0.3, STEPS, exact=True)
    assert np.array_equal(bits(s.get_u()), bits(ref["u"].ravel(order="F")))
    s.close()


def test_batch_of_cold_and_given_starts():
    """Members that start cold and from a given state run in one batch as
    they do alone."""
    from asetsmatlabmaxflow_gb300 import native as N

    ctx = N.Context.default()
    batch, members, alone = N.Batch(ctx), [], []
    for i, dims in enumerate([(40, 22, 10), (66, 15, 9), (24, 31, 12)]):
        ct, al, cs = _inputs("binary", dims, 1, 20 + i)
        if i == 2:
            ct[0, 0, 0] = np.inf
        pair = []
        for _ in range(2):
            s = N.Solver(ctx, "binary", dims)
            s.set_inputs(ct, al, cs)
            if i == 1:
                s.set_initial(np.full(dims, 0.5, np.float32), np.minimum(cs, ct), np.minimum(cs, ct))
            pair.append(s)
        batch.add(pair[0])
        members.append(pair[0])
        alone.append(pair[1])
    its = batch.run(40, 1e-4, 0.3, STEPS)
    for m, a, it in zip(members, alone, its):
        assert a.run(40, 1e-4, 0.3, STEPS) == it
        assert float(np.max(np.abs(m.get_u() - a.get_u()))) <= 1e-5
    batch.close()
