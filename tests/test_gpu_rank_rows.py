"""Rows put in order by counting (triplets, raw CSR, transposes) at the edges of that kernel:
64 rows and 2,048 entries a turn, rows of 127 to 129 entries (129 sort), with and without a
diagonal to insert, empty rows, rectangular shapes. Bit-exact against numpy: rows by stable
order of column, a missing diagonal as 0.0 at its place; transposes by stable order of row."""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


def _rows(n, m, lens, seed, diag):
    """Rows of lens[i] random columns (repeats allowed), diagonals kept out unless asked for."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n), lens)
    c = rng.integers(0, m, len(r))
    if not diag:
        c = np.where(c == r, (c + 1) % m, c)
    else:
        first = np.unique(r, return_index=True)[1]
        c[first] = np.minimum(r[first], m - 1)
    return r, c, rng.standard_normal(len(r))


CASES = {
    "one": (1, 3, [1]), "turn63": (63, 80, [7] * 63), "turn64": (64, 64, [32] * 64),
    "turn65": (65, 70, [31] * 65), "entries": (64, 500, [33] * 64),
    "long126": (70, 900, [3] * 40 + [126] + [0] * 29), "long127": (70, 900, [3] * 40 + [127] + [1] * 29),
    "long128": (70, 900, [128] * 70), "long129": (70, 900, [2] * 69 + [129]),
    "empty": (300, 310, [0, 5] * 150), "wide": (100, 3000, [20] * 100),
}


def _expected(n, r, c, v):
    miss = np.setdiff1d(np.arange(n), r[r == c])
    r, c, v = np.append(r, miss), np.append(c, miss), np.append(v, np.zeros(len(miss)))
    at = np.lexsort((c, r))  # stable
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return rp, c[at], v[at]


def _check(M, want):
    got = M.download()
    assert np.array_equal(got.rowPtr, want[0]) and np.array_equal(got.colInd, want[1])
    assert np.array_equal(got.values, want[2])


@pytest.mark.parametrize("diag", [False, True])
@pytest.mark.parametrize("name", CASES)
def test_rows_in_order(name, diag):
    from faspxx_b200 import capi, sol
    capi.init(0)
    n, m, lens = CASES[name]
    r, c, v = _rows(n, m, lens, len(name) + n, diag)
    want = _expected(n, r, c, v)
    for base in (0, 1):
        rp = np.zeros(n + 1, np.int64)
        np.cumsum(lens, out=rp[1:])
        _check(sol.MAT.FromCSRRaw(n, rp + base, c + base, v, mcol=m), want)
    at = np.random.default_rng(1).permutation(len(r))
    M = sol.MAT.FromCOO(n, m, r[at], c[at], v[at])
    _check(M, _expected(n, r[at], c[at], v[at]))
    A = M.download()
    rows = np.repeat(np.arange(n), np.diff(A.rowPtr.astype(np.int64)))
    k = np.lexsort((rows, A.colInd))
    tp = np.zeros(m + 1, np.int64)
    np.cumsum(np.bincount(A.colInd, minlength=m), out=tp[1:])
    _check(M.Transpose(), (tp, rows[k], A.values[k]))
