"""Triangles that collapse to a line at an iterate of the FP64 advancement, and at no time that the FP32 filter
looks at: a vertex lies on the line of a fixed edge, beyond its end, and the third corner crosses that line just
when the first step ends. The point-plane distance of such a triangle is rounding alone and may report a
contact, which tau_max, bit for bit the oracle's, has to keep."""
import numpy as np
import pytest

import rs_gb300 as R
import rs_oracle as O
from ccd_scenes import soup

pytestmark = pytest.mark.gpu


def scene(seed, x, gap, close_factor):
    """The vertex at distance x along the edge's line and a little above it; (faces, start, velocity, the time of
    the crossing)."""
    rng = np.random.default_rng(seed)
    th = rng.uniform(0.9, 1.2)
    d, m = np.array([np.cos(th), np.sin(th), 0.0]), np.array([np.sin(th), -np.cos(th), 0.0])
    a, b, p = np.zeros(3), d, x * d + [0.0, 0.0, 0.02]
    d0 = np.linalg.norm(p - b)
    t = (d0 - (gap if d0 > gap else close_factor * d0)) * (1.0 - 1e-12)  # the first step at speed 1
    c = rng.uniform(0.2, 0.8) * d + t * m
    far = np.array([0.0, 0.0, 5e3])  # long edges: one window
    f, s = soup([[a, b, c], [p, p + [0.0, 0.1, 3.0], p + [0.1, 0.0, 3.0]], [far, far + [1e3, 0, 0], far + [0, 1e3, 0]]])
    v = np.zeros((9, 3))
    v[2] = -m
    return f, s, v, t


@pytest.mark.parametrize("x,horizon,gap,close_factor", [(2.2, 60.0, 0.05, 0.5), (2.5, 60.0, 0.05, 0.5), (2.5, 60.0, 2.0, 0.5)])
def test_a_collapse_between_the_filters_times(x, horizon, gap, close_factor):
    met = 0
    for seed in range(400):
        f, p, v, t = scene(seed, x, gap, close_factor)
        kw = {"reference_length": 1.0, "gap": gap, "close_factor": close_factor}
        o = O.ccd_first_contact(f, p, v, horizon * t, **kw)
        g = R.CcdSurface(f, len(p)).first_contact(p, v, horizon * t, R.ccd_options(**kw))
        for k in ("tau_max", "contact", "windows", "pairs_tested", "close_pairs", "touching_pairs"):
            assert g[k] == o[k], (seed, k, o, g)
        met += o["contact"]
    assert met > 0  # some of the collapses are such contacts
