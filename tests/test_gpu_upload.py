"""What an upload finds out about a matrix on the device -- CheckCSR's verdict, diagonal
pointers, tile span, 16-bit reach, row classes -- against numpy, at the edges: tiles of 256
rows, chunks of 4,096 entries, the greatest class count, row length and table the class form
takes. Whole numbers: equal."""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from faspxx_b200 import capi, sol
    capi.init(0)
    return sol


def _csr(lens, cols, vals, mcol=None):
    rp = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    return P.CSRMatrix(len(lens), mcol or len(lens), rp.astype(np.uint32),
                       np.asarray(cols, np.uint32), np.asarray(vals, np.float64))


def _random(n, m, seed, longest=9, dense_row=0):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, longest, n)
    if dense_row:
        lens[n // 2] = dense_row
    lens[0] = max(lens[0], 1)
    return _csr(lens, rng.integers(0, m, lens.sum()), rng.standard_normal(lens.sum()), m)


def _diagonal_classes(classes, n):
    """n rows of one entry, `classes` different values."""
    return _csr(np.ones(n, int), np.arange(n), 1.0 + (np.arange(n) % classes))


def _row_of(length, n=2000):
    lens = np.ones(n, int)
    lens[5] = length
    cols = np.concatenate([np.arange(5), np.arange(length) + 5, np.arange(6, n)])
    return _csr(lens, cols, np.ones(len(cols)))


def _classes(A):
    """(classes, table entries) by the definition, 0, 0 where the form is not built."""
    if A.nnz / A.nrow > 16:
        return 0, 0
    seen, entries = set(), 0
    rp = A.rowPtr.astype(np.int64)
    bits = A.values.view(np.int64)
    for r in range(A.nrow):
        s = slice(rp[r], rp[r + 1])
        if s.stop - s.start > 64:
            return 0, 0
        key = (tuple(A.colInd[s].astype(np.int64) - r), tuple(bits[s]))
        if key not in seen:
            seen.add(key)
            entries += s.stop - s.start
            if len(seen) > 4096 or entries > max(64, A.nnz // 8):
                return 0, 0
    return len(seen), entries


CASES = {
    "one": _csr([1], [0], [2.0]),
    "rows255": _random(255, 255, 1), "rows256": _random(256, 300, 2), "rows257": _random(257, 200, 3),
    "chunk": _random(300, 9000, 4, dense_row=4096), "chunk+1": _random(300, 9000, 5, dense_row=4097),
    "long": _random(70, 70000, 6, dense_row=20000),
    "near": _csr([1, 1], [32767, 0], [1.0, 1.0], 40000), "far": _csr([1, 1], [32768, 0], [1.0, 1.0], 40000),
    "classes4096": _diagonal_classes(4096, 4096 * 8), "classes4097": _diagonal_classes(4097, 4097 * 8),
    "table": _diagonal_classes(1000, 8000), "table+1": _diagonal_classes(1000, 7999),
    "row64": _row_of(64), "row65": _row_of(65),
    "poisson3d": P.poisson3d(13, 11, 9), "poisson2d": P.poisson2d(65),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("device", [False, True])
def test_upload_facts(gpu, name, device):
    A = CASES[name]
    if device:
        import ctypes as C
        import torch
        from faspxx_b200.capi import check, lib
        d = [torch.from_numpy(a).cuda() for a in (A.rowPtr.view(np.int32), A.colInd.view(np.int32),
                                                  A.values)]
        h = C.c_void_p()  # no synchronisation: the upload waits for torch's stream
        check(lib.fasp_gpu_mat_create_device(A.nrow, A.mcol, A.nnz, *(t.data_ptr() for t in d),
                                             C.byref(h)), "MAT")
        M = gpu.MAT(_handle=h)
    else:
        M = gpu.MAT(A)
    B = M.download()
    assert np.array_equal(B.rowPtr, A.rowPtr) and np.array_equal(B.colInd, A.colInd)
    assert np.array_equal(B.values, A.values)
    assert np.array_equal(M.diag_ptr(), A.diag_ptr())
    rp = A.rowPtr.astype(np.int64)
    ends = np.append(rp[:-1:256], rp[-1])
    span = max((b + 3) // 4 * 4 - a // 4 * 4 for a, b in zip(ends[:-1], ends[1:]))
    assert M.TileInfo()[0] == span
    rows = np.repeat(np.arange(A.nrow), np.diff(rp))
    near = bool(np.all(np.abs(A.colInd.astype(np.int64) - rows) <= 32767))
    assert M.Col16Info()[0] == near
    assert M.RowClassInfo()[1:3] == _classes(A)
    if name.startswith("poisson"):
        assert M.RowClassInfo()[0] == 2 and M.RowClassInfo()[3] == (7 if "3d" in name else 5)


@pytest.mark.parametrize("what", ["first", "last", "order", "beyond", "column"])
def test_upload_rejects(gpu, what):
    from faspxx_b200 import capi
    A = P.poisson2d(40)
    rp, ci = A.rowPtr.copy(), A.colInd.copy()
    if what == "first":
        rp[0] = 1
    elif what == "last":
        rp[-1] -= 1
    elif what == "order":
        rp[700] = rp[690]
    elif what == "beyond":
        rp[700] = A.nnz + 1000
    else:
        ci[-1] = A.mcol
    with pytest.raises(capi.FaspError) as err:
        gpu.MAT(P.CSRMatrix(A.nrow, A.mcol, rp, ci, A.values))
    assert err.value.code == -17
