"""The hierarchical products at the sizes where their kernels change path: leaves of 1 to 8 rows
(each has its own lane mapping in the near field), trees of one leaf, of one bottom group and of
one to three levels of groups, empty far fields, batches across the three vectors of a pass, and
inputs far from one in magnitude (the channel grid's powers of two).

Tolerance 1e-6 of the largest entry against the FP64 oracle: a kernel value carries at most about
sixteen FP32 half-units (r^2 to the 5/3, the normal form, the weight), and on the smallest meshes
nothing averages them."""
import numpy as np
import pytest

import golden_io as G
import rs_oracle as O
import rs_gb300 as R
from rs_gb300 import generators as gen

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.fixture(scope="module")
def ctx():
    return R.Context(0)


def tetrahedron():
    P = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1.2]], float)
    return P, np.array([[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]], np.uint32)


MESHES = {
    "tetrahedron": tetrahedron,                                        # one leaf
    "icosahedron": lambda: gen.icosphere(0),                           # a few leaves, one group
    "torus-9x5": lambda: gen.noisy_torus(9, 5, 1.0, 0.4, 0.01, 3),     # 16 to 20 leaves: one or two groups
    "torus-41x13": lambda: gen.noisy_torus(41, 13, 1.0, 0.35, 0.004, 4),
    "torus-120x75": lambda: gen.noisy_torus(120, 75, 1.0, 0.3, 0.002, 5),  # over 128 bottom groups
}


def dual_areas(P, F):
    a, _, _ = O.face_geometry(P, F)
    return np.bincount(F.ravel().astype(np.int64), np.repeat(a / 3.0, 3), minlength=len(P))


@pytest.mark.parametrize("mesh,leaf_size,chi", [
    ("tetrahedron", 8, 0.5), ("tetrahedron", 1, 0.5), ("icosahedron", 8, 0.5), ("icosahedron", 2, 1.0),
    ("torus-9x5", 8, 0.0), ("torus-9x5", 5, 0.5),
    *[("torus-41x13", k, 0.5) for k in range(1, 9)],
    ("torus-120x75", 8, 0.5), ("torus-120x75", 3, 0.5), ("torus-120x75", 1, 0.5)])
def test_products_at_the_edges(ctx, mesh, leaf_size, chi):
    P, F = MESHES[mesh]()
    opts = R.ClusterTreeOptions(chi=chi, leaf_size=leaf_size)
    rng = np.random.default_rng(6)
    x = rng.standard_normal((4, 3 * len(P)))
    m = R.FaceMetricTree(F, P, R.Exponents(), opts, ctx)
    y = m.apply(x, 0.7, 0.3)
    yo = O.FaceMetricTree(P, F, chi=chi, leaf_size=leaf_size).apply(x, 0.7, 0.3)
    mass, tau = dual_areas(P, F), 2.0 - 5.0 / 3.0
    v = R.VertexFractionalTree(P, mass, tau, opts, ctx)
    z = v.apply(x)
    zo = O.VertexFractionalTree(P, mass, tau, chi=chi, leaf_size=leaf_size).apply(x)
    print(f"{mesh} leaf {leaf_size} chi {chi}: metric {G.normwise(y, yo):.1e} vertex {G.normwise(z, zo):.1e}")
    assert G.normwise(y, yo) <= TOL and G.normwise(z, zo) <= TOL
    # a vector alone, in a pair and in a pass of three gives the same bits
    for k in (1, 2, 3):
        assert np.array_equal(m.apply(x[:k], 0.7, 0.3), y[:k]) and np.array_equal(v.apply(x[:k]), z[:k])
    one = np.ones(3 * len(P))
    assert np.all(m.apply(one, 0.0, 1.0) == 0.0) and np.all(v.apply(one) == 0.0)


def test_products_scale_by_powers_of_two(ctx):
    """The channel grid follows the largest magnitude, so a power of two scales the result exactly
    while every FP32 part stays a normal number."""
    P, F = MESHES["torus-41x13"]()
    m = R.FaceMetricTree(F, P, R.Exponents(), R.ClusterTreeOptions(), ctx)
    x = np.random.default_rng(7).standard_normal(3 * len(P))
    y = m.apply(x)
    for k in (-40, -3, 5, 60):
        assert np.array_equal(m.apply(x * 2.0 ** k), y * 2.0 ** k), k
