"""Jacobi solves of small systems where nothing reads their norms, which run in one launch: as the
preconditioner of one CG iteration, x = alpha z with z = 40 sweeps on r = b from zero and
alpha = (z, r) / (A z, z), against numpy. (A Jacobi solver of its own reports norms and runs sweep by
sweep.)

Each sweep rounds a row of at most 127 products and adds to an iteration that contracts: z differs
by at most 40 x 130 ulp of max|z|; the three sums of n <= 1,024 terms by as many ulp. 3e-12 of
max|x| covers both; FP32 sweeps only precondition, and their solves are held to the FP64 residual.
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


def _system(n, twice=False):
    """Rows of up to 127 entries (n = 125: dense), off-diagonal ones stored twice with `twice`;
    symmetric, dominant."""
    rng = np.random.default_rng(n)
    D = rng.uniform(-1, 1, (n, n))
    if n > 125:
        D *= rng.random((n, n)) < 6.0 / n
        D[n // 2] = rng.uniform(-1, 1, n) * (rng.random(n) < 100.0 / n)
    D = D + D.T
    np.fill_diagonal(D, 0.0)
    np.fill_diagonal(D, 1.5 * np.abs(D).sum(1) + 1.0)
    rp, ci, va = [0], [], []
    for i in range(n):
        for j in np.nonzero(D[i])[0]:
            k = 2 if twice and j != i else 1
            ci += [j] * k
            va += [D[i, j] / k] * k
        rp.append(len(ci))
    return D, P.CSRMatrix(n, n, np.array(rp, np.uint32), np.array(ci, np.uint32), np.array(va))


def _sweeps(D, r, most, least, rel):
    z, w, done = np.zeros(len(r)), 0.8 / np.diag(D), 0
    first = None
    for it in range(most):
        res = r - D @ z
        if it >= least:
            first = np.linalg.norm(res) if first is None else first
            if np.linalg.norm(res) < rel * first:
                break
        z = z + res * w
        done += 1
    return z, done


@pytest.mark.parametrize("n,twice", [(1, False), (2, False), (31, False), (32, False), (32, True),
                                     (33, False), (125, False), (1024, False)])
@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("least", [40, 0, 3])
def test_preconditioner_in_one_launch(gpu, n, twice, lanes, least):
    D, A = _system(n, twice)
    assert A.nnz * 10 + n * 8 <= 200 * 1024  # fits the launch's shared memory
    b = np.random.default_rng(1).uniform(-1, 1, n)
    M = gpu.MAT(A)
    M.SetLanes(lanes)
    s = gpu.configure("cg", maxIter=1, minIter=1, relTol=0.0, absTol=0.0, pcd="jacobi", pcdWeight=0.8,
                      pcdIter=40, pcdMinIter=least, pcdRelTol=1e-3, pcdAbsTol=0.0)
    s.Setup(M)
    x = np.zeros(n)
    s.Solve(b, x)
    z, done = _sweeps(D, b, 40, least, 1e-3)
    assert done < 40 if least < 40 else done == 40  # the test on the device stops early
    want = z * (z @ b) / (z @ (D @ z))
    assert np.max(np.abs(x - want)) <= 3e-12 * np.max(np.abs(want))
    assert s.info.launches < 40  # a launch a sweep would be more


# one unknown is solved by half a BiCGStab step, whose other half then divides by zero, as the
# reference's does
@pytest.mark.parametrize("alg,n", [("bicgstab", 32), ("bicgstab", 33), ("bicgstab", 125),
                                   ("fgmres", 1), ("fgmres", 32), ("fgmres", 33), ("fgmres", 125)])
def test_fp32_sweeps_precondition(gpu, n, alg):
    from faspxx_b200 import capi
    D, A = _system(n)
    b = np.random.default_rng(2).uniform(-1, 1, n)
    its = []
    for prec in (capi.FP64, capi.MIXED):
        s = gpu.configure(alg, maxIter=200, relTol=1e-10, absTol=0.0, pcd="jacobi", pcdWeight=0.8,
                          pcdIter=3, pcdMinIter=3)
        s.SetPrecision(prec)
        s.Setup(gpu.MAT(A))
        x = np.zeros(n)
        assert s.Solve(b, x) == 0
        assert np.linalg.norm(b - D @ x) <= 1.01e-10 * np.linalg.norm(b)
        its.append(s.GetIterations())
    # each refinement step gains 1e-4 and starts a new space: three of them
    assert its[1] <= 3 * its[0] + 3
