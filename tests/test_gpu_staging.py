"""Host arrays of volumes with padded rows: the device memory kept to pad them
is bounded, and without any the copies give the same values."""
import numpy as np
import pytest

from tests.gpu_helpers import bits, require_gpu

pytestmark = pytest.mark.gpu


def _solve(N, ctx, dims, L):
    g = np.random.default_rng(2)
    ct, al = (np.asfortranarray((0.05 + g.random(dims + (L,))).astype(np.float32)) for _ in range(2))
    s = N.Solver(ctx, "potts", dims, L)
    s.set_inputs(ct, al)
    s.run(3, 0.0, 0.3, 0.11)
    out = [bits(s.get_u()), *(bits(f) for f in s.get_flows())]
    s.close()
    return out


@pytest.mark.parametrize("most", ["0", "1", "4096", "1000000"])
def test_any_staging_size_gives_the_same_values(monkeypatch, most):
    """No buffer (as where none can be had), rows longer than it, a few rows
    at a time, and out copies of several runs (above 4 MB)."""
    from asetsmatlabmaxflow_gb300 import native as N

    require_gpu()
    dims, L = (333, 61, 30), 2
    want = _solve(N, N.Context.default(), dims, L)
    monkeypatch.setenv("ASETS_STAGE_BYTES", most)
    ctx = N.Context()
    for a, b in zip(want, _solve(N, ctx, dims, L)):
        assert np.array_equal(a, b)
    ctx.close()


def test_staging_memory_is_bounded():
    import torch

    from asetsmatlabmaxflow_gb300 import native as N

    require_gpu()
    dims = (250, 330, 240)                     # 79 MB an array
    ct = np.ones(dims, np.float32, order="F")
    s = N.Solver(N.Context.default(), "binary", dims)
    before = torch.cuda.mem_get_info()[0]
    s.set_inputs(ct, ct, ct)
    assert before - torch.cuda.mem_get_info()[0] <= 40 << 20   # 32 MB, whole driver blocks
    s.close()
