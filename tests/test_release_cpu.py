"""Handles give their memory back only when the device they live on has nothing left to do, whatever
device the destroying thread has current. Pool memory can go to another handle at once, so a
product enqueued by an asynchronous call must have been waited for by then. On a runtime of two
devices without GPUs (fakecuda.py)."""
import ctypes as C

import numpy as np
import pytest

from faspxx_b200 import problems as P
from tests import fakecuda


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fakecuda.load(tmp_path_factory.mktemp("fake"))



def _matrix(lib):
    A, h = P.poisson2d(40), C.c_void_p()
    assert lib.fasp_gpu_mat_create(A.nrow, A.mcol, A.nnz, A.rowPtr.ctypes.data, A.colInd.ctypes.data,
                                   A.values.ctypes.data, C.byref(h)) == 0
    return A, h


def _device(lib, a):
    p = C.c_void_p()
    assert lib.fasp_gpu_malloc(C.byref(p), a.nbytes + 16) == 0
    assert lib.fasp_gpu_memcpy_h2d(p, a.ctypes.data, a.nbytes) == 0
    return p


def _product_in_flight(lib, A, h):
    x, y = _device(lib, np.ones(A.mcol)), _device(lib, np.ones(A.nrow))
    assert lib.fasp_gpu_mat_apply_async(h, x, y, lib.fake_stream()) == 0


@pytest.mark.parametrize("current", [1, 0])  # the device of the handles, and another one
@pytest.mark.parametrize("kind", ["matrix", "transposed", "solver", "setup again", "batch"])
def test_destroy_waits_for_the_handles_device(lib, kind, current):
    from faspxx_b200 import capi
    assert lib.fasp_gpu_init(1) == 0
    lib.fasp_gpu_synchronize()
    A, h = _matrix(lib)
    early = lib.fake_early_frees()
    if kind == "transposed":
        z = _device(lib, np.ones(A.mcol))
        assert lib.fasp_gpu_mat_mult_transpose_add_async(h, z, z, _device(lib, np.ones(A.mcol)),
                                                         lib.fake_stream()) == 0
    if kind in ("solver", "setup again"):
        cfg = capi.Config()
        lib.fasp_gpu_default_config(C.byref(cfg), capi.CG)
        s = C.c_void_p()
        assert lib.fasp_gpu_solver_create(C.byref(cfg), C.byref(s)) == 0
        assert lib.fasp_gpu_solver_setup(s, h) == 0
    if kind == "batch":
        bt = C.c_void_p()
        rows = _device(lib, np.array([0, 700, 1600], np.uint32))
        B = P.CSRMatrix(1600, 1600, np.arange(1601, dtype=np.uint32), np.arange(1600, dtype=np.uint32),
                        np.ones(1600))
        d = [_device(lib, a) for a in (B.rowPtr, B.colInd, B.values)]
        assert lib.fasp_gpu_batch_create(2, rows, B.nnz, *d, 1, C.byref(bt)) == 0
    assert lib.fake_early_frees() == early
    _product_in_flight(lib, A, h)
    lib.fake_use_device(current)
    if kind == "solver":
        assert lib.fasp_gpu_solver_destroy(s) == 0
    elif kind == "setup again":
        assert lib.fasp_gpu_solver_setup(s, h) == 0
    elif kind == "batch":
        assert lib.fasp_gpu_batch_destroy(bt) == 0
    else:
        assert lib.fasp_gpu_mat_destroy(h) == 0
    assert lib.fake_early_frees() == early
    assert lib.fake_device() == current


def _with_each_allocation_failing(lib, make, destroy):
    """make() once for every device allocation it does, that one failing (and its retry): the codes.
    Nothing that a failed call allocated stays, and nothing is released under unfinished work."""
    h = C.c_void_p()
    lib.fasp_gpu_synchronize()
    early = lib.fake_early_frees()
    assert make(h) == 0 and destroy(h) == 0  # contexts and page-locked blocks are in their lists
    blocks, codes = lib.fake_blocks(), []
    for k in range(100):
        failed = lib.fake_failures()
        lib.fake_fail_in(k)
        code = make(h)
        lib.fake_fail_in(-1)
        if lib.fake_failures() == failed:  # fewer than k allocations
            assert code == 0 and destroy(h) == 0
            break
        assert code in (0, -20), (k, code)
        if code == 0:
            assert destroy(h) == 0
        codes.append(code)
        assert lib.fake_blocks() <= blocks, k  # an idle context may have been given back
        assert make(h) == 0 and destroy(h) == 0
    assert len(codes) < 100
    assert lib.fake_early_frees() == early  # what was enqueued before a failure is waited for
    return codes


def test_batch_without_memory_for_slices(lib):
    """The resident kernels' copy of the matrix (columns, FP64 and FP32 values) is a convenience: a
    batch for which the device has no room left but for the matrix itself is solved without it."""
    assert lib.fasp_gpu_init(1) == 0
    n = 1600
    rows = _device(lib, np.array([0, 700, n], np.uint32))
    d = [_device(lib, a) for a in (np.arange(n + 1, dtype=np.uint32), np.arange(n, dtype=np.uint32),
                                   np.ones(n))]
    codes = _with_each_allocation_failing(
        lib, lambda h: lib.fasp_gpu_batch_create(2, rows, n, *d, 1, C.byref(h)),
        lib.fasp_gpu_batch_destroy)
    assert codes.count(0) == 3
    # a system too large for a cluster beside small ones: its vectors, too, come before the copy
    n = 66000
    rows = _device(lib, np.array([0, 65800, n], np.uint32))
    d = [_device(lib, a) for a in (np.arange(n + 1, dtype=np.uint32), np.arange(n, dtype=np.uint32),
                                   np.ones(n))]
    codes = _with_each_allocation_failing(
        lib, lambda h: lib.fasp_gpu_batch_create(2, rows, n, *d, 1, C.byref(h)),
        lib.fasp_gpu_batch_destroy)
    # the copy's three; nine vectors and the FP32 values of matrix and classes, for which there is
    # room without the copy
    assert codes.count(0) == 3 + 11


@pytest.mark.parametrize("what", ["transpose", "coo", "csr_raw", "create", "stencil"])
def test_matrices_without_memory(lib, what):
    """Every allocation on the way to a matrix may fail: the call says so and leaves nothing behind.
    Transposes and triplets, whose short rows travel as 16-byte records, do without the records
    where there is no memory for them (8-byte keys)."""
    assert lib.fasp_gpu_init(1) == 0
    A, h = _matrix(lib)
    rows = np.repeat(np.arange(A.nrow, dtype=np.uint32), np.diff(A.rowPtr.astype(np.int64)))
    zero, one = np.zeros(1, np.int32), np.ones(1)
    make = {
        "transpose": lambda t: lib.fasp_gpu_mat_transpose(h, C.byref(t)),
        "coo": lambda t: lib.fasp_gpu_mat_create_coo(A.nrow, A.mcol, A.nnz, rows.ctypes.data,
                                                     A.colInd.ctypes.data, A.values.ctypes.data, 0,
                                                     C.byref(t)),
        "csr_raw": lambda t: lib.fasp_gpu_mat_create_csr_raw(A.nrow, A.mcol, A.nnz,
                                                             A.rowPtr.ctypes.data,
                                                             A.colInd.ctypes.data,
                                                             A.values.ctypes.data, 0, C.byref(t)),
        "create": lambda t: lib.fasp_gpu_mat_create(A.nrow, A.mcol, A.nnz, A.rowPtr.ctypes.data,
                                                    A.colInd.ctypes.data, A.values.ctypes.data,
                                                    C.byref(t)),
        "stencil": lambda t: lib.fasp_gpu_mat_create_stencil(
            20, 20, 1, 1, zero.ctypes.data, zero.ctypes.data, zero.ctypes.data, one.ctypes.data,
            C.byref(t)),
    }[what]
    codes = _with_each_allocation_failing(lib, make, lib.fasp_gpu_mat_destroy)
    assert codes.count(0) == (1 if what in ("transpose", "coo") else 0)
    assert lib.fasp_gpu_mat_destroy(h) == 0


@pytest.mark.parametrize("precision", ["FP64", "MIXED", "MIXED_RELIABLE"])
def test_batch_without_room_for_clusters(lib, precision):
    """A device that holds no cluster of the resident kernels (a process limited to some SMs) solves
    the batch in global memory, as devices did before there were clusters; with room it does not."""
    from faspxx_b200 import capi
    assert lib.fasp_gpu_init(1) == 0
    n = 1600
    rows = _device(lib, np.array([0, 700, n], np.uint32))
    d = [_device(lib, a) for a in (np.arange(n + 1, dtype=np.uint32), np.arange(n, dtype=np.uint32),
                                   np.ones(n))]
    b, x = _device(lib, np.ones(n)), _device(lib, np.ones(n))
    bt = C.c_void_p()
    assert lib.fasp_gpu_batch_create(2, rows, n, *d, 1, C.byref(bt)) == 0
    try:
        for clusters in (16, 0, 16):
            lib.fake_set_clusters(clusters)
            lib.fake_clear_launches()
            refused = lib.fake_refused()
            # the fake device computes nothing; a refined solve stops at its first residual, 0
            code = lib.fasp_gpu_batch_solve(bt, b, x, 1e-8, 10, getattr(capi, precision), 1e-2,
                                            None, None)
            assert code == 0 and lib.fake_refused() == refused
            if precision != "MIXED":
                plain, resident = lib.fake_launches(b"batch_pcg"), lib.fake_launches(b"batch_resident")
                assert (plain, resident) == ((0, 1) if clusters else (1, 0))
    finally:
        lib.fake_set_clusters(16)
    assert lib.fasp_gpu_batch_destroy(bt) == 0


def _solver(lib, h, cfg):
    s = C.c_void_p()
    code = lib.fasp_gpu_solver_create(C.byref(cfg), C.byref(s))
    if code == 0:
        code = lib.fasp_gpu_solver_setup(s, h)
        assert lib.fasp_gpu_solver_destroy(s) == 0
    return code


@pytest.mark.parametrize("alg,more", [
    ("CG", {}), ("CG", {"pcd": 1}), ("CG", {"pcd": 2}), ("CG", {"precision": "MIXED"}),
    ("CG", {"persistent": 1}), ("CG", {"persistent": 2}), ("CG", {"pcd": 1, "precision": "MIXED_RELIABLE"}),
    ("BICGSTAB", {}), ("BICGSTAB", {"precision": "MIXED"}), ("BICGSTAB", {"precision": "MIXED_RELIABLE"}),
    ("GMRES", {}), ("GMRES", {"precision": "MIXED"}), ("FGMRES", {}), ("JACOBI", {}), ("MG", {})])
def test_setup_without_memory(lib, alg, more):
    """Every allocation of a solver's Setup may fail: the code says so, and nothing is left behind
    once the solver is destroyed."""
    from faspxx_b200 import capi
    assert lib.fasp_gpu_init(1) == 0
    A, h = _matrix(lib)
    cfg = capi.Config()
    lib.fasp_gpu_default_config(C.byref(cfg), getattr(capi, alg))
    cfg.prm.maxIter = 20
    cfg.pcdPrm.minIter = cfg.pcdPrm.maxIter = 1
    for k, v in more.items():
        setattr(cfg, k, getattr(capi, v) if isinstance(v, str) else v)
    codes = _with_each_allocation_failing(lib, lambda t: _solver(lib, h, cfg), lambda t: 0)
    assert codes and codes.count(0) == 0
    assert lib.fasp_gpu_mat_destroy(h) == 0
