"""The multigrid solve of the preconditioner at the sizes where its kernel changes path: fewer rows
than blocks, one level, one cluster of blocks for every batch width, a cluster for the narrow widths and
the whole grid for the wide ones, the grid for all.

A column's arithmetic (row sums, dot products, scalars) depends neither on the columns beside it nor on
which blocks hold its rows, so a batch gives each column's own result bit for bit, on whichever path it
goes; the narrow widths are compared with the oracle elsewhere. A zero column stays zero."""
import numpy as np
import pytest

import rs_gb300 as R
from rs_gb300 import generators as gen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return R.Context(0)


def tetrahedron():
    P = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1.2]], float)
    return P, np.array([[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]], np.uint32)


@pytest.mark.parametrize("mesh,vcycles", [
    ("tetrahedron", 1), ((9, 5), 6), ((20, 15), 1), ((33, 20), 6), ((66, 66), 2), ((75, 75), 6), ((100, 80), 6), ((140, 100), 3)])
def test_columns_do_not_depend_on_the_batch(ctx, mesh, vcycles):
    P, F = tetrahedron() if mesh == "tetrahedron" else gen.noisy_torus(*mesh, 1.0, 0.35, 0.002, 5)
    S = R.SaddleSolver(F, P, R.Exponents(), R.solver_options(vcycles=vcycles), ctx)
    r = np.random.default_rng(31).standard_normal((4, S.n))
    r[:, S.n_dofs:] = 0.0
    r[2, 0::3] = r[2, 1::3] = r[2, 2::3] = 0.0
    one = np.concatenate([S.precondition(r[k:k + 1]) for k in range(4)])
    assert np.isfinite(one).all() and not one[2].any()
    for nb in (2, 3, 4):
        assert np.array_equal(S.precondition(r[:nb]), one[:nb]), nb
    assert np.array_equal(S.precondition(r), S.precondition(r))
