"""A batch with members of all groups (binary and labelled, 2D and 3D), whose
launches are branches of one graph: every member's EXACT result is its lone
one, over runs repeated on the same batch and after a member has left early."""
import numpy as np
import pytest

from tests.gpu_helpers import bits, require_gpu

pytestmark = pytest.mark.gpu

MEMBERS = [("binary", (65, 49), 1), ("binary", (24, 21, 17), 1), ("potts", (40, 33), 3), ("ishikawa", (20, 18, 9), 4),
           ("binary", (33, 130), 1), ("potts", (17, 16, 12), 2)]


def test_members_of_every_group():
    require_gpu()
    from asetsmatlabmaxflow_gb300 import native as N

    ctx = N.Context.default()
    g = np.random.default_rng(8)
    b, solvers, lone = N.Batch(ctx), [], []
    for model, dims, L in MEMBERS:
        la = {"binary": (), "potts": (L,), "ishikawa": (L - 1,)}[model]
        ct = np.asfortranarray(g.random(dims + ((L,) if L > 1 else ())).astype(np.float32))
        al = np.asfortranarray((0.05 + 0.3 * g.random(dims + la)).astype(np.float32))
        cs = np.asfortranarray(g.random(dims).astype(np.float32)) if model == "binary" else None
        pair = []
        for _ in range(2):
            s = N.Solver(ctx, model, dims, L)
            s.set_inputs(ct, al, cs)
            pair.append(s)
        it = pair[0].run(70, 2e-4, 0.3, 0.11, exact=True)
        lone.append((it, pair[0].get_u()))
        pair[0].close()
        b.add(pair[1])
        solvers.append(pair[1])
    for _ in range(2):
        its = b.run(70, 2e-4, 0.3, 0.11, exact=True)
        for s, it, (ref_it, u) in zip(solvers, its, lone):
            assert it == ref_it
            np.testing.assert_array_equal(bits(s.get_u()), bits(u))
    b.close()
    for s in solvers:
        s.close()
