"""The interaction lists where their test changes its arithmetic: leaf and node boxes are compared in FP32
with a margin, in FP64 inside the margin and where theta or the mesh's extent leaves FP32's range. The
lists equal the oracle's, entry for entry: separation ratios on both sides of theta^2 and equal to
it (a grid of equal boxes at whole distances), meshes far from the origin, tiny and huge ones."""
import numpy as np
import pytest

import rs_oracle as O
import rs_gb300 as R
from rs_gb300 import generators as gen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return R.Context(0)


def boxes_on_a_grid(m):
    """m^3 equal tetrahedra at the points of a grid: the separations repeat exactly."""
    T = np.array([[0, 0, 0], [0.25, 0, 0], [0, 0.25, 0], [0, 0, 0.25]])
    c = np.stack(np.meshgrid(*[np.arange(m, dtype=float)] * 3, indexing="ij"), -1).reshape(-1, 3)
    P = (c[:, None] + T[None]).reshape(-1, 3)
    f = np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]])
    return P, (f[None] + 4 * np.arange(len(c))[:, None, None]).reshape(-1, 3).astype(np.uint32)


def torus():
    return gen.noisy_torus(64, 48, 1.0, 0.35, 0.004, 4)


MESHES = {
    "torus": (torus, 1.0, 0.0), "far": (torus, 1.0, 1e5), "tiny": (torus, 1e-9, 0.0), "huge": (torus, 1e9, 3e9),
    "grid": (lambda: boxes_on_a_grid(10), 1.0, 0.0),
}


@pytest.mark.parametrize("mesh,theta,leaf", [
    ("torus", 0.25, 8), ("torus", 0.5, 4), ("torus", 1e-5, 8), ("torus", 1e-7, 8), ("torus", 3e6, 8), ("torus", 1.0, 1),
    ("far", 0.3, 8), ("tiny", 0.25, 8), ("huge", 0.25, 8), ("grid", 0.25, 4), ("grid", 0.5, 4), ("grid", 0.125, 4)])
def test_lists_equal_the_oracles(ctx, mesh, theta, leaf):
    make, scale, offset = MESHES[mesh]
    P, F = make()
    P = scale * P + offset
    t = R.BhTree.build(F, P, R.BhOptions(theta, leaf), ctx)
    o = O.BhTree(P, F, theta=theta, leaf_size=leaf)
    lists, ol = t.export()[1], o.lists()
    for k in ("lumped_off", "lumped", "exact_off", "exact"):
        assert np.array_equal(lists[k], ol[k]), k
