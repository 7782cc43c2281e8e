"""Rows of very different lengths through the device-side inspection of a matrix and the conversion of
raw CSR arrays: long rows are looked at by a whole block, short ones by a thread. Diagonal pointers,
bandwidth, errors and converted arrays against numpy; and the time of a matrix of a few long rows
against that of the same number of entries in many short ones."""
import time

import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sol():
    from faspxx_b200 import capi, sol
    capi.init(0)
    return sol


def _mat(n, mcol, lens, seed=0, near=None):
    rng = np.random.default_rng(seed)
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(lens)
    rows = np.repeat(np.arange(n), lens)
    ci = rng.integers(0, mcol, rp[-1]) if near is None else \
        np.clip(rows + rng.integers(-near, near + 1, rp[-1]), 0, mcol - 1)
    return P.CSRMatrix(n, mcol, rp.astype(np.uint32), ci.astype(np.uint32),
                       rng.uniform(-1, 1, rp[-1]))


def _first_diag(A):
    rows = np.repeat(np.arange(A.nrow), np.diff(A.rowPtr.astype(np.int64)))
    out = np.zeros(A.nrow, np.uint32)
    at = np.nonzero(A.colInd == rows)[0][::-1]
    out[rows[at]] = at  # the first of several wins
    return out


LENS = {
    "edge": [127, 128, 129, 0, 130, 1] * 50,                 # on both sides of the limit
    "chunks": [4095, 4096, 4097, 5, 8192, 129, 1, 12289] * 6,  # ends on and off the 4,096-entry chunks
    "all long": [300] * 600,                                  # every row of every tile
    "one": [20000],
    "mixed": [3] * 255 + [50000] + [2] * 256 + [1000, 3] * 200,  # last row of a tile, an all-short tile
}


@pytest.mark.parametrize("name", sorted(LENS))
@pytest.mark.parametrize("near", [None, 60])
def test_diagonal_and_reach(sol, name, near):
    lens = np.array(LENS[name])
    n = len(lens)
    A = _mat(n, max(n, 70000) if near is None else n, lens, n, near)
    M = sol.MAT(A)
    assert np.array_equal(M.diag_ptr(), _first_diag(A))
    rows = np.repeat(np.arange(n, dtype=np.int64), lens)
    assert bool(M.Col16Info()[0]) == bool(np.all(np.abs(A.colInd - rows) <= 32767))
    x, y = np.random.default_rng(1).uniform(-1, 1, A.mcol), sol.DVec(n)
    M.Apply(sol.DVec.from_numpy(x), y)
    terms = A.values * x[A.colInd]
    want = np.array([terms[a:b].sum() for a, b in zip(A.rowPtr[:-1], A.rowPtr[1:])])
    scale = np.array([np.abs(terms[a:b]).sum() for a, b in zip(A.rowPtr[:-1], A.rowPtr[1:])])
    assert np.all(np.abs(y.numpy() - want) <= 2.3e-16 * (lens + 2) * 2 * scale)


@pytest.mark.parametrize("at", [0, 128, 5000, 19999])
@pytest.mark.parametrize("raw", [False, True])
def test_bad_column_in_a_long_row(sol, at, raw):
    from faspxx_b200 import capi
    A = _mat(3, 30000, np.array([2, 20000, 2]))
    A.colInd[2 + at] = 30000
    with pytest.raises(capi.FaspError) as e:
        sol.MAT.FromCSRRaw(A.nrow, A.rowPtr, A.colInd, A.values, mcol=30000) if raw else sol.MAT(A)
    assert e.value.code == -17


@pytest.mark.parametrize("name", sorted(LENS))
@pytest.mark.parametrize("base", [0, 1])
def test_raw_csr(sol, name, base):
    """Columns ascending in each row, equal ones in input order, a missing diagonal as an explicit 0."""
    lens = np.array(LENS[name])
    n = len(lens)
    A = _mat(n, max(n, 3000), lens, 7)
    M = sol.MAT.FromCSRRaw(n, A.rowPtr + np.uint32(base), A.colInd + np.uint32(base), A.values,
                           mcol=A.mcol).download()
    rows = np.repeat(np.arange(n), lens)
    lack = np.setdiff1d(np.arange(n), rows[A.colInd == rows])
    r, c = np.concatenate([rows, lack]), np.concatenate([A.colInd.astype(np.int64), lack])
    v = np.concatenate([A.values, np.zeros(len(lack))])
    o = np.lexsort((np.arange(len(r)), c, r))
    assert np.array_equal(M.rowPtr, np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]))
    assert np.array_equal(M.colInd, c[o]) and np.array_equal(M.values, v[o])


@pytest.mark.parametrize("raw", [False, True])
def test_few_long_rows_take_no_longer(sol, raw):
    """64 rows of 200,000 entries against 200,000 of 64, the better of three each. The two move the
    same bytes; one thread a row took some seven times as long. A factor of two leaves room for a
    busy host, and another two for the conversion, which sorts long rows and ranks short ones."""
    def best(A):
        t = []
        for _ in range(3):
            t0 = time.perf_counter()
            M = sol.MAT.FromCSRRaw(A.nrow, A.rowPtr, A.colInd, A.values, mcol=A.mcol) if raw \
                else sol.MAT(A)
            t.append(time.perf_counter() - t0)
            del M
        return min(t)

    wide, tall = (P.CSRMatrix(n, 200_000, np.arange(0, n * k + 1, k, dtype=np.uint32),
                              np.tile(np.arange(k, dtype=np.uint32) * (200_000 // k), n),
                              np.ones(n * k)) for n, k in ((64, 200_000), (200_000, 64)))
    assert best(wide) <= (4 if raw else 2) * best(tall)
