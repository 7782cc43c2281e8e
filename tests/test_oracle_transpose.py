"""The oracle's transpose is there whether or not the reference is built on this machine, and is the
transpose: entries of a column in the order of their rows."""
import numpy as np
import pytest

from faspxx_b200 import problems as P


@pytest.mark.parametrize("kind", ["port", "ref"])
@pytest.mark.parametrize("A", [P.convdiff3d(5, 1.0), P.poisson2d(7, 3)])
def test_transpose(oracle_built, kind, A):
    rp, ci, va, dp = oracle_built.transpose(kind, A)
    T = A.scipy().T.tocsr()
    T.sort_indices()
    assert np.array_equal(rp, T.indptr) and np.array_equal(ci, T.indices)
    assert np.array_equal(va, T.data)
    assert np.array_equal(ci[dp], np.arange(A.nrow))
