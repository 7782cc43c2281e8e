"""Batches at the ends of the on-chip kernels' range: with one right-hand side a cluster of eight
blocks holds 65,536 rows (a block's arrays hold threads * 8 / nrhs values, FP32 as FP64), where the
16-bit columns and the division of a column by the rows of a block reach their greatest values; one
row more runs in global memory. Every system's true residual meets the tolerance."""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


def _arrow(n, seed):
    """Tridiagonal, with a few entries to the far end of the system in both directions; symmetric."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    i = np.arange(n - 1)
    j = rng.integers(0, n, 400)
    rows = np.concatenate([i, j[j != n - 1 - j]])
    cols = np.concatenate([i + 1, n - 1 - j[j != n - 1 - j]])
    S = sp.coo_matrix((-rng.uniform(0.2, 1.0, len(rows)), (rows, cols)), shape=(n, n)).tocsr()
    S = S + S.T
    S = (S + sp.diags(np.asarray(abs(S).sum(1)).ravel() + rng.uniform(0.05, 0.1, n))).tocsr()
    S.sort_indices()
    return S, P.CSRMatrix(n, n, S.indptr.astype(np.uint32), S.indices.astype(np.uint32), S.data)


@pytest.mark.parametrize("nrhs,sizes", [(1, [32769, 65535, 65536, 65537]), (2, [32768, 32769]),
                                        (1, [65536, 7, 32768, 1])])
@pytest.mark.parametrize("precision", ["FP64", "MIXED", "MIXED_RELIABLE"])
def test_largest_on_chip(nrhs, sizes, precision):
    from faspxx_b200 import batch as BT, capi
    capi.init(0)
    made = [_arrow(n, n) if n > 7 else (None, P.poisson2d(n, 1, shift=0.5)) for n in sizes]
    B = BT.Batch([m for _, m in made], nrhs=nrhs)
    b = np.random.default_rng(7).standard_normal((nrhs, B.N))
    x = B.solve(b, relTol=1e-8, precision=getattr(capi, precision), innerRelTol=1e-2)[0]
    for (_, m), r0, r1 in zip(made, B.sys_row[:-1], B.sys_row[1:]):
        for k in range(nrhs):
            r = b[k, r0:r1] - m.matvec(x[k, r0:r1])
            # the FP64 recursive residual drifts from the true one by rounding only
            assert np.linalg.norm(r) <= 1.5e-8 * np.linalg.norm(b[k, r0:r1]), (m.nrow, k)
