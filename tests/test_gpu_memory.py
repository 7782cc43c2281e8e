"""The library's memory pool and its lists of idle contexts (faspxx_b200/csrc/mem.cu): what is given
back, what is taken again, and several threads at once."""
import ctypes as C
import gc
import threading

import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sol():
    from faspxx_b200 import capi, sol
    capi.init(0)
    return sol


def _large(n=8_000_000):
    """Three entries a row, about 0.5 GB on the device."""
    ci = np.minimum(np.arange(n, dtype=np.int64)[:, None] + np.arange(3)[None, :], n - 1)
    return P.CSRMatrix(n, n, np.arange(0, 3 * n + 1, 3, dtype=np.uint32),
                       ci.ravel().astype(np.uint32), np.random.default_rng(0).uniform(1, 2, 3 * n))


def test_trim_gives_idle_memory_back(sol):
    torch = pytest.importorskip("torch")
    A = _large()
    sol.MAT(P.poisson2d(8))  # the library's first allocations
    gc.collect()
    sol.trim()
    before = torch.cuda.mem_get_info(0)[0]
    M = sol.MAT(A)
    assert torch.cuda.mem_get_info(0)[0] < before - (400 << 20)
    del M
    gc.collect()
    sol.trim()
    # pieces that live allocations of this process hold may stay: 64 MB
    assert torch.cuda.mem_get_info(0)[0] >= before - (64 << 20)
    # and the library goes on
    x, y = sol.DVec.from_numpy(np.ones(A.mcol)), sol.DVec(A.nrow)
    sol.MAT(A).Apply(x, y)
    assert np.allclose(y.numpy(), A.matvec(np.ones(A.mcol)), rtol=1e-13, atol=0)


def test_idle_memory_is_bounded(sol):
    """Six matrices of about 1 GB each, destroyed: 4 GiB of them may wait for the next handles."""
    torch = pytest.importorskip("torch")
    A = _large(20_000_000)
    gc.collect()
    sol.trim()
    before = torch.cuda.mem_get_info(0)[0]
    held = [sol.MAT(A) for _ in range(6)]
    taken = before - torch.cuda.mem_get_info(0)[0]
    assert taken > 5 << 30
    del held
    gc.collect()
    kept = before - torch.cuda.mem_get_info(0)[0]
    assert kept <= (4 << 30) + (256 << 20)
    # the next one takes from there, and is right
    M = sol.MAT(A)
    x = np.random.default_rng(1).uniform(-1, 1, A.mcol)
    assert np.allclose(_apply(sol, M, A, x), A.matvec(x), rtol=1e-13, atol=1e-13)
    assert before - torch.cuda.mem_get_info(0)[0] <= kept + (512 << 20)
    del M
    gc.collect()
    sol.trim()
    assert torch.cuda.mem_get_info(0)[0] >= before - (64 << 20)


def _apply(sol, M, A, x):
    y = sol.DVec(A.nrow)
    M.Apply(sol.DVec.from_numpy(x), y)
    return y.numpy()


def test_destroyed_behind_an_asynchronous_product(sol):
    """A matrix destroyed right after its product was enqueued, and its memory taken at once by
    matrices of other values: the product has read its own."""
    torch = pytest.importorskip("torch")
    from faspxx_b200 import capi
    A = P.vardiff3d(60, np.random.default_rng(3).uniform(0.5, 2.0, (60, 60, 60)))
    B = P.CSRMatrix(A.nrow, A.mcol, A.rowPtr, A.colInd, -A.values)
    x = np.random.default_rng(4).uniform(-1, 1, A.mcol)
    want = _apply(sol, sol.MAT(A), A, x)
    stream = torch.cuda.Stream()
    dx = sol.DVec.from_numpy(x)
    for _ in range(10):
        y = [sol.DVec(A.nrow) for _ in range(4)]
        M = sol.MAT(A)
        for v in y:
            capi.check(capi.lib.fasp_gpu_mat_apply_async(M.h, dx.ptr, v.ptr,
                                                         C.c_void_p(stream.cuda_stream)), "apply")
        del M
        others = [sol.MAT(B) for _ in range(3)]
        stream.synchronize()
        for v in y:
            assert np.array_equal(v.numpy(), want)
        del others


def test_a_context_is_as_new_for_the_next_handle(sol):
    """Solvers and matrices one after another on the same contexts, with results that do not depend
    on what ran on them before: an abandoned solve, another size, a product."""
    A, B = P.poisson2d(30), P.poisson3d(9)
    b = np.random.default_rng(5).uniform(-1, 1, A.nrow)

    def solve(mat, rhs, iters):
        s = sol.configure("cg", maxIter=iters, relTol=1e-10, absTol=0.0, pcd="jacobi", pcdIter=1)
        s.Setup(sol.MAT(mat))
        x = np.zeros(mat.nrow)
        code = s.Solve(rhs, x)
        return code, s.GetIterations(), s.info.launches, x

    first = solve(A, b, 500)
    for _ in range(3):
        solve(B, np.ones(B.nrow), 3)  # ends at maxIter
        _apply(sol, sol.MAT(B), B, np.ones(B.nrow))
        gc.collect()
        again = solve(A, b, 500)
        assert again[:3] == first[:3] and np.array_equal(again[3], first[3])


def test_threads(sol):
    """Handles built, used and destroyed by several threads at once, each with its own matrices."""
    wrong = []

    def work(k):
        rng = np.random.default_rng(k)
        for _ in range(20):
            n = int(rng.integers(4, 40))
            A = P.vardiff3d(n, rng.uniform(0.5, 2.0, (n, n, n)))
            x = rng.uniform(-1, 1, A.mcol)
            M = sol.MAT(A)
            T = M.Transpose()
            y, z = _apply(sol, M, A, x), _apply(sol, T, A, x)
            want, scale = A.matvec(x), np.max(np.abs(A.values)) * 7 * 1e-15
            if np.max(np.abs(y - want)) > scale or np.max(np.abs(z - A.scipy().T @ x)) > scale:
                wrong.append((k, n))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
