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
