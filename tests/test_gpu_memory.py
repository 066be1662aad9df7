"""Device memory that a 3D solver takes: arrays that are in use at different
times share their place."""
import pytest

from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


# inputs, flows in two parities, then binary: gradient source, pt and u in two;
# Potts: source (and pt), divergence, u and ps in two
@pytest.mark.parametrize("model,L,arrays", [("binary", 1, 3 + 6 + 6), ("potts", 3, 8 * 3 + 4 * 3 + 2)])
def test_arrays_of_a_solver(model, L, arrays):
    import torch

    from asetsmatlabmaxflow_gb300 import native as N

    require_gpu()
    dims = (256, 128, 128)   # 16 MB an array, whole blocks of the driver
    ctx = N.Context.default()
    before = torch.cuda.mem_get_info()[0]
    s = N.Solver(ctx, model, dims, L)
    taken = before - torch.cuda.mem_get_info()[0]
    s.close()
    one = 256 * 128 * 128 * 4
    assert taken <= arrays * one + one // 2
