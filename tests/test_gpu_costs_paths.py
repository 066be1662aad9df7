"""Cost terms and contrast weights on the paths that sizes and alignment
choose: 16-byte and single accesses, warps' edges, short axes, device arrays
off 16 bytes, degenerate images."""
import numpy as np
import pytest

from oracle import costs as C
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


def _img(shape, seed):
    return np.asfortranarray((np.random.default_rng(seed).random(shape) * 700.0 - 120.0).astype(np.float32))


# rows either side of one and of 32 lanes of one and of four rows, columns
# either side of a block's eight, planes either side of a block's sixteen
@pytest.mark.parametrize("shape", [(128, 8, 16), (129, 9, 17), (132, 7, 15), (124, 1, 33), (32, 16, 1),
                                   (33, 17, 2), (4, 3, 40), (1, 5, 7), (1, 1, 1), (260, 10, 3)])
@pytest.mark.parametrize("squared", [False, True])
def test_alpha_shapes(shape, squared):
    from asetsmatlabmaxflow_gb300 import costs

    img = _img(shape, 1)
    got = costs.alpha_contrast(img, 0.05, 0.3, 10.0, squared=squared, labels=2)
    with np.errstate(invalid="ignore"):
        ref = C.alpha_contrast(img, 0.05, 0.3, 10.0, squared=squared)
    for l in range(2):
        # differences of float data over the range: 4 half-ulps of the
        # gradient, times c = 10 and b = 0.3 in the exponential's argument
        np.testing.assert_allclose(got[..., l], ref, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_device_arrays_off_16_bytes(offset):
    import torch

    from asetsmatlabmaxflow_gb300 import native as N

    shape, L = (64, 9, 5), 3
    img = _img(shape, 2)
    n = img.size
    scr = np.random.default_rng(3).integers(-1, L + 2, size=n).astype(np.int32)
    scr[:L] = np.arange(1, L + 1)
    flat = torch.from_numpy(img.ravel(order="F").copy())
    d = torch.zeros(n + offset, device="cuda")[offset:].copy_(flat)
    s = torch.zeros(n + offset, dtype=torch.int32, device="cuda")[offset:].copy_(torch.from_numpy(scr))
    out = torch.zeros(n * L + offset, device="cuda")[offset:]
    al = torch.zeros(n * L + offset, device="cuda")[offset:]
    torch.cuda.synchronize()
    ctx = N.Context.default()
    counts = np.zeros(L * 256, np.uint32)
    N.check(N.lib().asets_cost_histogram_ll(ctx.handle, N.DEVICE, d.data_ptr(), s.data_ptr(), n, L, 1e-10,
                                            out.data_ptr(), counts.ctypes.data))
    ref, cref = C.cost_histogram_ll(img, scr.reshape(shape, order="F"), L)
    assert np.array_equal(counts.reshape(L, 256).astype(np.int64), cref)
    assert np.array_equal(out.cpu().numpy(), ref.ravel(order="F"))
    N.check(N.lib().asets_alpha_contrast(ctx.handle, N.DEVICE, d.data_ptr(), *shape, 1, 0.0, 0.2, 10.0, 0, L,
                                         al.data_ptr()))
    a = C.alpha_contrast(img, 0.0, 0.2, 10.0).ravel(order="F")
    np.testing.assert_allclose(al.cpu().numpy(), np.tile(a, L), rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("L", [1, 5, 32])
def test_histogram_of_many_voxels(L):
    from asetsmatlabmaxflow_gb300 import costs

    shape = (117, 90, 31)
    img = _img(shape, 5)
    scr = np.asfortranarray(np.random.default_rng(6).integers(0, L + 1, size=shape).astype(np.int32))
    ct, counts = costs.histogram_ll(img, scr, L)
    ref, cref = C.cost_histogram_ll(img, scr, L)
    assert np.array_equal(counts.astype(np.int64), cref) and np.array_equal(ct, ref)


def test_degenerate_images():
    """A constant image has no range (0/0), a raw one needs none; a tiny range
    still scales; not-a-number voxels stay local."""
    from asetsmatlabmaxflow_gb300 import costs

    flat = np.full((8, 6, 4), 3.0, np.float32, order="F")
    assert np.all(np.isnan(costs.alpha_contrast(flat)))
    assert np.all(costs.alpha_contrast(flat, 0.1, 0.2, normalize=False) == np.float32(0.1) + np.float32(0.2))
    tiny = _img((8, 8, 4), 7) * np.float32(1e-42)
    with np.errstate(all="ignore"):
        np.testing.assert_allclose(costs.alpha_contrast(tiny), C.alpha_contrast(tiny, 0.0, 0.2, 10.0),
                                   rtol=1e-5, atol=1e-6)
    img = _img((9, 9, 9), 8)
    img[4, 4, 4] = np.nan
    got = costs.alpha_contrast(img, 0.0, 0.2, 1.0)
    assert np.isnan(got).sum() == 6 and not np.isnan(got[4, 4, 4])
