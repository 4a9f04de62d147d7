"""The collision cap where its FP32 decisions end: slivers, near-degenerate and parallel edges, tiny, huge and
far-away scenes, gaps down to FP32's resolution, few iterations, several windows, resting pairs,
many pairs left for the FP64 advancement. tau_max is the oracle's bit for bit, the counts are
equal."""
import numpy as np
import pytest

import ccd_scenes as S
import rs_gb300 as R
import rs_oracle as O

pytestmark = pytest.mark.gpu

KEYS = ("tau_max", "contact", "windows", "pairs_tested", "close_pairs", "touching_pairs")


def same(f, p, v, tau_end, ell, **kw):
    o = O.ccd_first_contact(f, p, v, tau_end, reference_length=ell, **kw)
    g = R.CcdSurface(f, len(p)).first_contact(p, v, tau_end, R.ccd_options(reference_length=ell, **kw))
    assert {k: g[k] for k in KEYS} == {k: o[k] for k in KEYS}, (o, g)
    assert g["evaluations"] >= g["pairs_tested"]
    return g


@pytest.mark.parametrize("scale,offset", [(1e-3, 0.0), (1e-12, 0.0), (1e-25, 0.0), (1e15, 0.0), (1.0, 1e4), (1e-3, 50.0)])
def test_scales_and_offsets(scale, offset):
    for seed in range(6):
        f, p, v, tau_end, ell = S.random_soup(300 + seed)
        same(f, scale * p + offset, scale * v, tau_end, scale * ell)
    f, p, v, tau_end, ell = S.torus_sweep(24, 12, reach=3.0)
    same(f, scale * p + offset, scale * v, tau_end, scale * ell)


@pytest.mark.parametrize("width", [1e-2, 1e-4, 1e-6, 1e-9, 0.0])
def test_slivers_and_parallel_edges(width):
    rng = np.random.default_rng(7)
    tris = []
    for _ in range(60):  # needles of that width, many of them parallel to an axis
        a = rng.standard_normal(3)
        d = np.eye(3)[rng.integers(3)] if rng.random() < 0.5 else rng.standard_normal(3)
        tris.append([a, a + d, a + 0.5 * d + width * rng.standard_normal(3)])
    f, p = S.soup(tris)
    v = np.repeat(rng.standard_normal((60, 3)), 3, 0)
    same(f, p, v, 1.0, 1.0)
    same(f, p, 0.0 * v, 1.0, 1.0)


@pytest.mark.parametrize("kw", [{"gap": 1e-7}, {"gap": 1e-4}, {"gap": 1.5}, {"max_iterations": 1}, {"max_iterations": 3},
                                {"max_iterations": 400}, {"close_factor": 0.99}])
def test_options(kw):
    for reach in (0.5, 6.0):
        same(*S.torus_sweep(36, 18, reach=reach), **kw)


def test_many_pairs_left():
    """A cloud of triangles closing in on itself: thousands of pairs are near their contact."""
    rng = np.random.default_rng(3)
    c = rng.uniform(-1.0, 1.0, (700, 1, 3))
    f, p = S.soup(c + 0.12 * rng.standard_normal((700, 3, 3)))
    v = np.repeat(-c[:, 0], 3, 0) + 0.05 * rng.standard_normal((2100, 3))
    same(f, p, v, 0.3, 0.5, gap=0.3)
    same(f, p, v, 0.3, 0.5, gap=0.01)
