"""The energy where its passes change path: trees of one block of 32 leaves (climbed in shared memory
alone), of one leaf more and of several blocks; few work items (four warps share one) and just more than
that; leaves of one face to eight; the fast and the general exponents, with and without the
differential.

The comparison, with its tolerances, is the one of test_bh_gpu: lists equal, energy and differential
against the FP64 oracle."""
import numpy as np
import pytest

import rs_gb300 as R
from rs_gb300 import generators as gen
from test_bh_gpu import check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return R.Context(0)


def tetrahedron():
    P = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1.2]], float)
    return P, np.array([[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]], np.uint32)


MESHES = {"tetrahedron": tetrahedron, "icosahedron": lambda: gen.icosphere(0),
          **{f"torus-{a}x{b}": (lambda a=a, b=b: gen.noisy_torus(a, b, 1.0, 0.4, 0.004, 3))
             for a, b in ((8, 8), (12, 8), (20, 12), (48, 34), (56, 40), (64, 48))}}


@pytest.mark.parametrize("exponents", [(6.0, 12.0), (4.5, 9.0)])
@pytest.mark.parametrize("mesh,theta,leaf", [
    ("tetrahedron", 0.5, 8), ("tetrahedron", 0.5, 1), ("icosahedron", 0.25, 3), ("torus-8x8", 0.5, 8), ("torus-8x8", 0.5, 4),
    ("torus-12x8", 0.5, 6), ("torus-20x12", 0.0, 8), ("torus-48x34", 0.25, 8), ("torus-56x40", 0.25, 8), ("torus-64x48", 0.5, 8),
    ("torus-64x48", 0.5, 5)])
def test_energy_at_the_edges(ctx, mesh, theta, leaf, exponents):
    P, F = MESHES[mesh]()
    ex = R.Exponents(*exponents)
    t, _, E, dE = check(ctx, P, F, theta, *exponents, leaf=leaf)
    assert abs(t.try_energy(ex) - E) <= 1e-12 * abs(E)
    t.refit(P)  # from the state the first left
    E2, dE2 = t.energy_and_differential(ex)
    assert E2 == E and np.array_equal(dE2, dE)
