"""getm_tridiagonal on column counts and levels at the edges of its blocks (32 columns) and of its
load batches (4 levels): FP64, the oracle's expressions in its order, so the tolerance is 0."""
import numpy as np
import pytest

import oracle
from code_b200.getm import Context
from code_b200.grid import Grid
from helpers import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [1, 31, 32, 33, 300])
@pytest.mark.parametrize("kmax,fi,lt", [(1, 0, 1), (3, 1, 3), (4, 0, 4), (5, 1, 4), (8, 1, 8), (9, 0, 9), (60, 1, 60),
                                        (150, 0, 150)])
def test_tridiagonal_edges(ncol, kmax, fi, lt):
    rng = np.random.default_rng(ncol + kmax)
    g = Grid(4, 4, kmax, 1.0, 1.0)
    au, cu = -rng.random((kmax + 1, ncol)), -rng.random((kmax + 1, ncol))
    bu, du = 1.5 - au - cu, rng.normal(size=(kmax + 1, ncol))
    want = np.full((kmax + 1, ncol), 7.0)
    o = oracle.Oracle(g)
    for q in range(ncol):
        col = [np.ascontiguousarray(a[:, q]) for a in (au, bu, cu, du)]
        want[fi:lt + 1, q] = o.tridiagonal(kmax, fi, lt, *col)[fi:lt + 1]
    value = dev(np.full((kmax + 1, ncol), 7.0))
    Context(g).tridiagonal(kmax, fi, lt, *[dev(a) for a in (au, bu, cu, du)], value)
    assert np.array_equal(host(value), want)
