"""The shape autotuner of a batch times the candidates only where one of them can matter: for
systems that are too large to be solved on chip."""
import numpy as np
import pytest

from faspxx_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,solves", [([8, 20, 33], 2), ([8, 260], 12)])
def test_autotune_times_what_depends_on_the_shape(sizes, solves):
    from faspxx_b200 import batch as BT, capi
    capi.init(0)
    B = BT.Batch([P.poisson2d(m, shift=0.5) for m in sizes], nrhs=1)
    done = []
    solve = B.solve
    B.solve = lambda *a, **k: done.append(B.shape) or solve(*a, **k)
    shape, ms = B.autotune(np.ones((1, B.N)), reps=2)
    assert len(done) == solves and shape in BT.SHAPES and 0 < ms < float("inf")
    assert shape == B.shape and (solves > 2 or set(done) == {shape})
