"""The batch kernels that keep a system's vectors on chip, at the edges of their size classes
(blocks of 256, 512 and 1,024 threads, clusters of 2, 4 and 8, and systems too large for them) and
with columns in every block of a cluster. Each right-hand side meets the stop test (relative
residual below relTol, times 1.5 for the recursive residual's drift, as in test_gpu_batch), which
on these matrices (eigenvalues in [0.3, 6]) bounds the error; FP64 iterations are the oracle's
CG's within max(2, 3%)."""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


def _system(n, seed):
    """Symmetric, diagonally dominant: a band, and couplings between far rows."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    i = np.arange(n - 1)
    f = rng.integers(0, n, (2, n // 3 + 1))
    r, c = np.concatenate([i, f[0]]), np.concatenate([i + 1, f[1]])
    keep = r != c
    r, c = r[keep], c[keep]
    S = sp.coo_matrix((-rng.uniform(0.2, 1.0, len(r)), (r, c)), shape=(n, n))
    S = (S + S.T).tocsr()
    S = (S + sp.diags(-np.asarray(S.sum(1)).ravel() + rng.uniform(0.3, 0.6, n))).tocsr()
    S.sort_indices()
    return P.CSRMatrix(n, n, S.indptr.astype(np.uint32), S.indices.astype(np.uint32), S.data)


def _check(sizes, nrhs, precision, relTol, oracle):
    from faspxx_b200 import batch as BT
    mats = [_system(n, n + k) for k, n in enumerate(sizes)]
    B = BT.Batch(mats, nrhs=nrhs)
    b = np.random.default_rng(nrhs).standard_normal((nrhs, B.N))
    x, it, rr, _ = B.solve(b, relTol=relTol, precision=precision, innerRelTol=1e-2)
    for k, m in enumerate(mats):
        s = slice(int(B.sys_row[k]), int(B.sys_row[k + 1]))
        S = m.scipy()
        for j in range(nrhs):
            res = np.linalg.norm(b[j, s] - S @ x[j, s]) / np.linalg.norm(b[j, s])
            assert res <= 1.5 * relTol, (m.nrow, j, res)
        if oracle and m.nrow <= 2100:
            from oracle import oracle as O
            ref = O.solve("port", m, "cg", b[0, s], np.zeros(m.nrow), maxIter=5000, minIter=0,
                          relTol=relTol, absTol=0.0, pcd="jacobi", pcdWeight=1.0, pcdIter=1)
            assert abs(int(it[k, 0]) - ref.iters) <= max(2, 0.03 * ref.iters)
    again = B.solve(b, relTol=relTol, precision=precision, innerRelTol=1e-2)
    assert np.array_equal(x, again[0]) and np.array_equal(it, again[1])


# rows a cluster holds: 64 bytes a thread and array, so threads * 8 / nrhs doubles a block
# (threads * 16 / nrhs floats), times the cluster
@pytest.mark.parametrize("nrhs,sizes", [
    (4, [2, 31, 32, 33, 511, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097]),
    (4, [8192, 8193, 16384, 16385]),
    (3, [64, 2049, 4100, 8200, 16390]),
    (2, [1023, 1025, 2049, 4097, 8193, 16385, 32769]),
    (1, [2047, 2049, 4097, 8193, 16385]),
])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "reliable"])
def test_size_classes(nrhs, sizes, precision):
    from faspxx_b200 import capi
    capi.init(0)
    p = {"fp64": capi.FP64, "mixed": capi.MIXED, "reliable": capi.MIXED_RELIABLE}[precision]
    _check(sizes, nrhs, p, 1e-10 if precision == "fp64" else 1e-8, precision == "fp64")


def test_one_long_row_runs_unsliced():
    """A dense row among short ones: padding its slice would double the matrix."""
    import scipy.sparse as sp
    from faspxx_b200 import batch as BT, capi
    capi.init(0)
    n = 400
    S = sp.identity(n, format="lil") * 3.0
    S[0, :] = -1.0 / n
    S[:, 0] = -1.0 / n
    S[0, 0] = 3.0
    S = S.tocsr()
    m = P.CSRMatrix(n, n, S.indptr.astype(np.uint32), S.indices.astype(np.uint32), S.data)
    B = BT.Batch([m, _system(50, 1)], nrhs=2)
    b = np.random.default_rng(0).standard_normal((2, B.N))
    for p in (capi.FP64, capi.MIXED_RELIABLE):
        x = B.solve(b, relTol=1e-8, precision=p, innerRelTol=1e-2)[0]
        for j in range(2):
            r = b[j, :n] - S @ x[j, :n]
            assert np.linalg.norm(r) <= 1.5e-8 * np.linalg.norm(b[j, :n])
