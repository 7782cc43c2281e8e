"""FP64 CG and BiCGStab on seven-point stencil masks, whose product kernels walk the planes of the grid
where an item gets at least three of them: the first iterations against the same solver with two
lanes a row, which gathers from plain CSR.

Both form every row and every sum from the same values; they differ in the order of summation.
A sum over 1e6 entries moves by less than 1e-13 of the sum of its terms, and cancellation in
s = r - alpha t and r = s - omega t (at most tenfold each on these diagonally dominant matrices)
carries that through four iterations: 1e-9 of a residual norm, 1e-11 of max|x|.
"""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from faspxx_b200 import capi, sol
    capi.init(0)
    return sol


def _matrix(shape, cut, symmetric):
    c = [-1.0, -1.2, -1.4, 10.0, -0.6, -0.8, -1.0]
    if symmetric:
        c[4:] = c[2::-1]
    A = P._from_stencil(shape, P._OFF3D, lambda k: c[k])
    n = A.nrow - cut  # the last plane loses its end
    rows = np.repeat(np.arange(A.nrow), np.diff(A.rowPtr.astype(np.int64)))
    keep = (rows < n) & (A.colInd < n)
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(np.bincount(rows[keep], minlength=n))
    return P.CSRMatrix(n, n, rp, A.colInd[keep], A.values[keep])


@pytest.mark.parametrize("alg", ["bicgstab", "cg"])
@pytest.mark.parametrize("pcd", [None, "jacobi"])
@pytest.mark.parametrize("shape,cut", [
    ((7, 43, 1800), 0),     # one column segment, most of it empty
    ((2, 300, 900), 0),     # the smallest S1; segments of 512 and 88 columns
    ((7, 43, 1801), 13),    # a ragged last plane
    ((101, 101, 101), 0),   # odd: no 16-byte groups
    ((96, 96, 96), 0),      # aligned
    ((128, 32, 300), 0),    # aligned, whole warps a plane
    ((256, 20, 220), 5),    # the largest S1
    ((257, 20, 220), 0),    # too wide to walk
    ((64, 90, 20), 0),      # too few planes an item
    ((33, 33, 33), 0)])
def test_first_iterations(gpu, shape, cut, pcd, alg):
    A = _matrix(shape, cut, alg == "cg")
    rng = np.random.default_rng(A.nrow)
    b, x0 = rng.uniform(-1, 1, A.nrow), rng.uniform(-1, 1, A.nrow)
    got = []
    for lanes in (1, 2):
        M = gpu.MAT(A)
        M.SetLanes(lanes)
        s = gpu.configure(alg, maxIter=4, relTol=1e-30, absTol=0.0, pcd=pcd,
                          pcdWeight=2.0 / 3.0, pcdIter=1)
        s.Setup(M)
        x = x0.copy()
        s.Solve(b, x)
        assert s.GetIterations() == 4
        got.append((x, s.History()[:5]))
    (x1, h1), (x2, h2) = got
    assert np.all(np.abs(h1 - h2) <= 1e-9 * h2)
    assert np.max(np.abs(x1 - x2)) <= 1e-11 * np.max(np.abs(x2))
