"""The multigrid solve on hierarchies whose coarsest level has fewer rows than the blocks of a cluster, so
that some blocks own none of it: surfaces of separate fans, each of which becomes one coarse row.

One right-hand side takes the cluster, several take the whole grid; a column's arithmetic depends on neither,
so both give it the same bits."""
import numpy as np
import pytest

import rs_gb300 as R

pytestmark = pytest.mark.gpu

CLUSTER = 16  # blocks


@pytest.fixture(scope="module")
def ctx():
    return R.Context(0)


def fans(m, k):
    """m disks, 3 apart: a hub and k rim vertices that alternate in height."""
    a = 2.0 * np.pi * np.arange(k) / k
    one = np.vstack([np.zeros((1, 3)), np.c_[np.cos(a), np.sin(a), 0.5 * (-1.0) ** np.arange(k)]])
    i = np.arange(k)
    face = np.c_[0 * i, 1 + i, 1 + (i + 1) % k]
    P = np.concatenate([one + [3.0 * s, 0.0, 0.0] for s in range(m)])
    return P, np.concatenate([face + s * (k + 1) for s in range(m)]).astype(np.uint32)


@pytest.mark.parametrize("per_component", [0, 1])
@pytest.mark.parametrize("m,k", [(15, 20), (13, 24), (11, 28), (10, 30), (9, 34), (7, 44), (6, 50), (5, 60)])
def test_fewer_coarse_rows_than_blocks(ctx, m, k, per_component):
    P, F = fans(m, k)
    S = R.SaddleSolver(F, P, R.Exponents(), R.solver_options(barycenter_per_component=per_component), ctx)
    levels = S.multigrid_levels()
    assert len(levels) == 2 and levels[-1][0] == m < CLUSTER
    r = np.random.default_rng(m).standard_normal((4, S.n))
    r[:, S.n_dofs:] = 0.0
    r[2] = 0.0
    one = np.concatenate([S.precondition(r[q:q + 1]) for q in range(4)])
    assert np.isfinite(one).all() and not one[2].any()
    for nb in (2, 3, 4):
        assert np.array_equal(S.precondition(r[:nb]), one[:nb]), nb


def test_more_columns_than_the_widest_batch(ctx):
    P, F = fans(5, 60)
    S = R.SaddleSolver(F, P, R.Exponents(), R.solver_options(coarse=0), ctx)
    with pytest.raises(R.RsError) as e:
        S.precondition(np.zeros((5, S.n)))
    assert (e.value.kind, e.value.operation, e.value.detail) == ("Internal", "preconditioner", "at most 12 multigrid columns")
