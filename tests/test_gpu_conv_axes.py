"""Convolutions whose tiles run along x or along z, by the volume's shape: the
same sums in the same order, so the transposed volume's bits, and the oracle's
values."""
import numpy as np
import pytest

from tests.gpu_helpers import require_gpu
from tests.test_gpu_conv import _bf16, conv_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(17, 1, 9), (33, 2, 16), (16, 15, 8), (1, 1, 40), (40, 3, 7), (3, 40, 7)])
@pytest.mark.parametrize("flip", [False, True])
def test_thin_volumes(shape, flip):
    import torch

    from asetsmatlabmaxflow_gb300 import native as N

    require_gpu()
    nz, nx, ny = shape
    g = np.random.default_rng(sum(shape))
    xt, x64 = _bf16(g.standard_normal((nz, nx, ny, 16)))
    wt, w64 = _bf16(0.2 * g.standard_normal((27, 16, 16)))
    bias = g.standard_normal(16).astype(np.float32)
    dx, dw, db = xt.cuda(), wt.cuda(), torch.from_numpy(bias).cuda()
    out = torch.full((nz, nx, ny, 16), float("nan"), device="cuda")
    torch.cuda.synchronize()
    N.check(N.lib().asets_conv3d_bf16(N.Context.default().handle, dx.data_ptr(), dw.data_ptr(), db.data_ptr(), None,
                                      out.data_ptr(), ny, nx, nz, 0, 1, int(flip)))
    err = np.abs(out.cpu().numpy() - conv_ref(x64, w64, bias, flip))
    # 433 roundings of at most 2^-23 of the sum of the terms' sizes
    assert (err <= 433 * 2.0 ** -23 * conv_ref(np.abs(x64), np.abs(w64), np.abs(bias), flip)).all()


@pytest.mark.parametrize("dims", [(20, 2, 37), (9, 1, 64)])
def test_network_gradients_along_z(dims):
    """Loss and gradients of a thin volume against the float64 oracle: BF16
    activations and gradients (2^-9 each, through four layers)."""
    from tests.test_gpu_conv_tiles import test_network_gradients_of_cut_tiles

    require_gpu()
    test_network_gradients_of_cut_tiles(dims)
