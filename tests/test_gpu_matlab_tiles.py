"""The Matlab-semantics solvers at the edges of their tiles (32 rows x 8
columns; in single precision binary 3D 64 rows x 12 to 16 columns), for label
counts with and without their own kernel, and with flows at, below and above
capacity: u bit for bit against the numpy restatement."""
import numpy as np
import pytest

from oracle import mtwin as M
from tests.gpu_helpers import require_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    require_gpu()


def _bits(a):
    a = np.ascontiguousarray(a)
    return a.view(np.uint64 if a.dtype == np.float64 else np.uint32)


def _run(model, shape, L, dtype, seed, its=25, cc=0.3, lo=0.02, hi=0.4):
    from asetsmatlabmaxflow_gb300 import matlab

    g = np.random.default_rng(seed)
    d3 = len(shape) == 3
    steps = 0.11 if d3 else 0.16
    lab = () if model == "binary" else (L,)
    ct = g.random(shape + lab).astype(dtype)
    al = (lo + (hi - lo) * g.random(shape + lab) ** 3).astype(dtype)
    pars = [*shape, *lab, its, 1e-30, cc, steps]
    dim = "3D" if d3 else "2D"
    if model == "binary":
        cs = g.random(shape).astype(dtype)
        return (getattr(matlab, "asetsBinaryMF" + dim)(cs, ct, al, pars),
                M.binary(cs, ct, al, its, 1e-30, cc, steps))
    ref = M.potts if model == "potts" else M.ishikawa
    name = "asetsPotts" if model == "potts" else "asetsIshikawa"
    return getattr(matlab, name + dim)(ct, al, pars), ref(ct, al, its, 1e-30, cc, steps)


def _check(got, ref, dtype):
    assert got[2] == ref[2] and got[0].dtype == dtype
    assert np.array_equal(_bits(got[0]), _bits(ref[0]))
    rt = 1e-12 if dtype == np.float64 else 2e-6
    assert np.allclose(got[1][:, 0].astype(np.float64), ref[1].astype(np.float64), rtol=rt, atol=0)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(32, 8), (33, 9), (31, 7), (1, 17), (65, 1), (40, 24),
                                   (32, 8, 3), (33, 9, 2), (64, 14, 4), (65, 15, 1), (3, 30, 9)])
@pytest.mark.parametrize("model,L", [("binary", 1), ("potts", 1), ("potts", 4), ("potts", 7),
                                     ("ishikawa", 2), ("ishikawa", 5)])
def test_tile_edges(model, L, shape, dtype):
    _check(*_run(model, shape, L, dtype, 1), dtype)


@pytest.mark.parametrize("cc", [0.25, 1.0 / 3.0, 2.0 ** 0.5, np.nextafter(0.5, 0), 3e-3, 7.0])
@pytest.mark.parametrize("model,L", [("binary", 1), ("potts", 3)])
def test_divisors(model, L, cc):
    """u/cc is formed from the reciprocal in double: divisors that are a power
    of two, ordinary, and with a significand of ones."""
    _check(*_run(model, (37, 21), L, np.float64, 3, cc=float(cc)), np.float64)
    _check(*_run(model, (9, 10, 6), L, np.float32, 4, cc=float(cc)), np.float32)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("lo,hi", [(1e-6, 2e-6), (5.0, 9.0), (0.0, 1e-30)])
def test_capacity_extremes(lo, hi, dtype):
    """Every cell at capacity, none, and capacities around zero."""
    _check(*_run("potts", (35, 18), 3, dtype, 5, lo=lo, hi=hi), dtype)
    _check(*_run("binary", (35, 18, 5), 1, dtype, 6, lo=lo, hi=hi), dtype)


# 32 x 8, 32 x 4 or 16 x 8 tiles by the tiles there are per SM (152) and the rows
# past the last: either side of one tile an SM and of four, cut in rows and columns
@pytest.mark.parametrize("shape", [(64, 600), (64, 615), (33, 9, 37), (33, 13, 40), (41, 1217), (41, 1209), (29, 30, 20)])
@pytest.mark.parametrize("model,L", [("binary", 1), ("potts", 3), ("potts", 7), ("ishikawa", 4)])
def test_tile_width_in_double(model, L, shape):
    _check(*_run(model, shape, L, np.float64, 7, its=8), np.float64)
