"""The weight gradients of five layers in one launch: no longer chains of
single-precision additions than a layer alone has over all SMs."""
import ctypes
import math
import subprocess
from pathlib import Path

import pytest

from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layers_lib(tmp_path_factory):
    from asetsmatlabmaxflow_gb300 import build

    require_gpu()
    src = Path(__file__).resolve().parent / "cuda" / "wgrad_layers_check.cu"
    out = tmp_path_factory.mktemp("wgradlayers") / "liblayers.so"
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, f"-I{build.CSRC}", f"-I{build.INCLUDE}",
                    "-shared", "-o", str(out), str(src), "-lcuda"], check=True)
    lib = ctypes.CDLL(str(out))
    lib.wgrad_layers_check.argtypes = [ctypes.c_int] * 3 + [ctypes.POINTER(ctypes.c_double)]
    return lib


@pytest.mark.parametrize("dims", [(112, 72, 64), (32, 60, 61), (48, 9, 3), (7, 2, 1)])
def test_error_of_the_sums(layers_lib, dims):
    """An accumulator takes the rows of one CTA in 150, 16 voxels an addition
    of at most an ulp (2^-23); then the sums of 5 sets and 30 CTAs at half an ulp each."""
    ny, nx, nz = dims
    worst = ctypes.c_double(1.0)
    assert layers_lib.wgrad_layers_check(ny, nx, nz, ctypes.byref(worst)) == 0
    steps = math.ceil(math.ceil(nx * nz / 30) / 5) * math.ceil(ny / 16)
    assert worst.value <= (steps + 35 / 2) * 2.0 ** -23
