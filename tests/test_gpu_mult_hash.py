"""MAT::Mult's hash rows at their edges: candidates per row around the size classes (64, 512,
2,048; 2,049 sorts) and around a warp's 32, R rows of one or several entries, few columns
(every lane of a warp adds to the same ones) and many. Bit-exact against the oracle."""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu

LENGTHS = {"class0": [0, 1, 31, 32, 33, 63, 64], "class1": [65, 64, 511, 512, 0],
           "class2": [513, 512, 2047, 2048, 3], "sorted": [2049, 64, 1]}


def _rows(rng, lens, m):
    rp = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    va = rng.standard_normal(rp[-1])
    va[::7] = -0.0
    return P.CSRMatrix(len(lens), m, rp.astype(np.uint32),
                       rng.integers(0, m, rp[-1]).astype(np.uint32), va)


@pytest.mark.parametrize("cols", [1, 7, 6000])
@pytest.mark.parametrize("each", [1, 5])
@pytest.mark.parametrize("name", LENGTHS)
def test_hash_rows(name, each, cols):
    from faspxx_b200 import capi, sol
    from oracle import oracle as O
    capi.init(0)
    rng = np.random.default_rng(cols + each)
    lens = np.array(LENGTHS[name] * 3)
    L = _rows(rng, lens // each if each > 1 else lens, 900)
    R = _rows(rng, np.full(900, each), cols)
    got = sol.MAT(L).Mult(sol.MAT(R)).download()
    for a, b in zip((got.rowPtr, got.colInd, got.values), O.mat_mult("port", L, R)):
        assert np.array_equal(a, b)
    assert np.array_equal(np.signbit(got.values), np.signbit(O.mat_mult("port", L, R)[2]))
