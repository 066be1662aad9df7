"""The 8 x 16-voxel convolution tiles, the weight-gradient rows of at most 112
voxels and the five-layer weight-gradient launch where a tile is cut: volumes
narrower than a tile, one voxel past it, rows that end within a K step."""
import ctypes

import numpy as np
import pytest

from oracle import wsnet as W
from tests.gpu_helpers import require_gpu
from tests.test_gpu_conv import _bf16, conv_ref, wgrad_lib  # noqa: F401
from tests.test_gpu_wsnet import _sample, _to_net_layout

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 9), (1, 15, 8), (3, 16, 7), (2, 17, 17), (1, 33, 40)])
def test_convolution_tiles(shape):
    """Sums of 432 products and a bias in FP32: 433 roundings of at most 2^-23
    of the sum of the terms' sizes."""
    import torch

    from asetsmatlabmaxflow_gb300 import native as N

    nz, nx, ny = shape
    g = np.random.default_rng(sum(shape))
    xt, x64 = _bf16(g.standard_normal((nz, nx, ny, 16)))
    wt, w64 = _bf16(0.2 * g.standard_normal((27, 16, 16)))
    bias = g.standard_normal(16).astype(np.float32)
    dx, dw, db = xt.cuda(), wt.cuda(), torch.from_numpy(bias).cuda()
    for flip in (False, True):
        out = torch.full((nz, nx, ny, 16), float("nan"), device="cuda")
        torch.cuda.synchronize()
        N.check(N.lib().asets_conv3d_bf16(N.Context.default().handle, dx.data_ptr(), dw.data_ptr(),
                                          db.data_ptr(), None, out.data_ptr(), ny, nx, nz, 0, 1, int(flip)))
        err = np.abs(out.cpu().numpy() - conv_ref(x64, w64, bias, flip))
        tol = 433 * 2.0 ** -23 * conv_ref(np.abs(x64), np.abs(w64), np.abs(bias), flip)
        assert (err <= tol).all()


@pytest.mark.parametrize("hp", [0, 1])
@pytest.mark.parametrize("dims", [(1, 1, 1), (15, 2, 3), (17, 3, 2), (112, 2, 2), (113, 2, 1), (225, 1, 3)])
def test_weight_gradient_rows(wgrad_lib, dims, hp):  # noqa: F811
    """FP32 sums over the voxels against double: a rounding of at most 2^-23 of
    the sum of the terms' sizes for each voxel and each CTA's partial."""
    worst = ctypes.c_double(1.0)
    assert wgrad_lib.wgrad_check(*dims, hp, ctypes.byref(worst)) == 0
    assert worst.value <= (np.prod(dims) + 152) * 2.0 ** -23


@pytest.mark.parametrize("dims", [(20, 17, 5), (9, 3, 6), (120, 2, 2)])
def test_network_gradients_of_cut_tiles(dims):
    """Loss and gradients against the float64 oracle; BF16 activations and
    gradients (2^-9 each, through four layers) stay within 2e-2 of a block's norm."""
    import torch

    from asetsmatlabmaxflow_gb300 import native as N

    L = 4
    net = N.WarmStartNet(N.Context.default(), nlab=L, seed=5)
    params = net.get_params()
    params += np.random.default_rng(2).normal(0, 0.02, params.size).astype(np.float32)
    net.set_params(params)
    host = _sample(dims, L, 4)
    dev = [torch.from_numpy(a).cuda() for a in host]
    torch.cuda.synchronize()
    loss, g = net.gradients(dims, *dev)
    x, tgt = _to_net_layout(dims, L, *host)
    loss_ref, g_ref, _ = W.loss_and_grads(params, x, tgt, L)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    for b in range(W.BLOCKS):
        base = b * (W.NW + 16)
        for part in (slice(base, base + W.NW), slice(base + W.NW, base + W.NW + 16)):
            r = g_ref[part]
            assert np.linalg.norm(g[part] - r) <= 2e-2 * max(np.linalg.norm(r), 1e-30)
    net.close()
