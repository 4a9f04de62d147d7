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


@pytest.mark.parametrize("mesh", [(66, 66), (140, 100)])
def test_two_threads_solve_at_once(mesh):
    """Two contexts, a thread each: their solves (each a kernel whose blocks wait for one another) run beside
    one another on the device and give what they give alone."""
    import threading

    P, F = gen.noisy_torus(*mesh, 1.0, 0.35, 0.002, 5)
    S = [R.SaddleSolver(F, P, R.Exponents(), R.solver_options(), R.Context(0)) for _ in range(2)]
    r = np.random.default_rng(9).standard_normal((3, S[0].n))
    r[:, S[0].n_dofs:] = 0.0
    want = {nb: S[0].precondition(r[:nb]) for nb in (1, 3)}
    bad = []

    def work(i):
        for k in range(40):
            nb = 1 if (i + k) % 2 else 3
            if not np.array_equal(S[i].precondition(r[:nb]), want[nb]):
                bad.append((i, k))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
