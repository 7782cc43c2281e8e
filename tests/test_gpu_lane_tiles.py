"""Products of FP64 matrices on four lanes a row whose entries stream through block tiles (more than
50 MB of entries, mean rows of 20 to 28): the bits of the lane kernels, which run the same rows in a
matrix below that size. Both take lane l's entries l, l + 4, ... with one FMA each and the same
shuffle tree, so MAT::Apply and MAT::Residual are equal bit for bit."""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [200_000, 200_001, 200_063])  # whole and partial last tiles of 64
@pytest.mark.parametrize("zero", [False, True])
def test_tiles_give_the_lane_kernels_bits(n, zero):
    from faspxx_b200 import capi, sol
    capi.init(0)
    rng = np.random.default_rng(n)
    lens = np.full(n, 24)
    lens[rng.integers(0, n, 2000)] = 0           # empty rows
    at = rng.integers(0, n // 64 - 1, 500) * 64  # a tile at the stage's limit
    lens[at] += 16
    lens[-1] = 3
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(lens)
    A = P.CSRMatrix(n, n, rp, rng.integers(0, n, rp[-1]).astype(np.uint32),
                    rng.uniform(-1, 1, rp[-1]))
    assert A.nnz * 12 > 50 << 20 and A.nnz >= 20 * n
    x = np.full(n, 1e-21) if zero else rng.uniform(-1, 1, n)  # below CLOSE_ZERO: r = b
    b = rng.uniform(-1, 1, n)

    def products(B, bb):
        M = sol.MAT(B)
        M.SetRowClass(0)
        M.SetLanes(4)
        y, r = sol.DVec(B.nrow), sol.DVec(B.nrow)
        dx = sol.DVec.from_numpy(x)
        M.Apply(dx, y)
        M.Residual(sol.DVec.from_numpy(bb), dx, r)
        return y.numpy(), r.numpy()

    y, r = products(A, b)
    for r0, r1 in ((0, 70_000), (70_000, 140_000), (140_000, n)):  # below 50 MB each
        p0, p1 = int(rp[r0]), int(rp[r1])
        assert (p1 - p0) * 12 < 50 << 20
        S = P.CSRMatrix(r1 - r0, n, (rp[r0:r1 + 1] - rp[r0]).astype(np.uint32), A.colInd[p0:p1],
                        A.values[p0:p1])
        ys, rs = products(S, b[r0:r1])
        assert np.array_equal(y[r0:r1], ys) and np.array_equal(r[r0:r1], rs)
    if zero:
        assert np.array_equal(r, b)
    assert sol.tile_timeouts() == 0
