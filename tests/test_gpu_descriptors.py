"""One resident solver whose launches find other tensor maps at the same
address from run to run: fast and EXACT, cold and warm starts, other tile
configurations.  Each run equals that of a solver made for it, bit for bit."""
import numpy as np
import pytest

from tests.gpu_helpers import bits, require_gpu

pytestmark = pytest.mark.gpu


def _run(s, warm, exact, tile):
    s.set_initial(*(warm or ()))
    s.run(6, 0.0, 0.35, 0.11, exact=exact, tile_config=tile)
    return bits(s.get_u())


@pytest.mark.parametrize("dims", [(70, 33, 21), (130, 97)])
def test_alternating_variants(dims):
    from asetsmatlabmaxflow_gb300 import native as N

    require_gpu()
    g = np.random.default_rng(4)
    cs, ct, al = (np.asfortranarray((0.05 + g.random(dims)).astype(np.float32)) for _ in range(3))
    ctx = N.Context.default()
    least = np.asfortranarray(np.minimum(cs, ct))
    warm = (np.full(dims, 0.5, np.float32, order="F"), least, least)
    plan = [(w, e, t) for t in (0, 1, 2, 3) for e in (False, True) for w in (None, warm)]
    want = []
    for p in plan:
        one = N.Solver(ctx, "binary", dims)
        one.set_inputs(ct, al, cs)
        want.append(_run(one, *p))
        one.close()
    s = N.Solver(ctx, "binary", dims)
    s.set_inputs(ct, al, cs)
    for _ in range(3):
        for p, u in zip(plan, want):
            assert np.array_equal(_run(s, *p), u), p[1:]
    s.close()
