"""The learned correction's kernels where their loads change: hubs of degree 3 and 70, vertex counts at and
off the multiples of a block and of a step of the weight gradient, against the plain PyTorch
reference and within the tolerances of test_learned_gpu."""
import numpy as np
import pytest

import rs_gb300 as R
from rs_gb300 import generators as gen
from test_learned_gpu import one_ring, reference, static_features

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def fan(m):
    """A closed surface with two hubs of degree m."""
    a = 2.0 * np.pi * np.arange(m) / m
    P = np.vstack([np.c_[np.cos(a), np.sin(a), 0.1 * np.cos(5 * a)], [[0, 0, 1.0], [0, 0, -1.0]]])
    i = np.arange(m)
    j = (i + 1) % m
    return P, np.vstack([np.c_[i, j, 0 * i + m], np.c_[j, i, 0 * i + m + 1]]).astype(np.uint32)


MESHES = {"fan3": lambda: fan(3), "fan70": lambda: fan(70), "torus-64": lambda: gen.noisy_torus(8, 8, 1.0, 0.4, 0.01, 2),
          "torus-1027": lambda: gen.noisy_torus(79, 13, 1.0, 0.35, 0.002, 3),
          "torus-1920": lambda: gen.noisy_torus(48, 40, 1.0, 0.35, 0.002, 3)}


@pytest.mark.parametrize("mesh", list(MESHES))
def test_forward_and_gradient(mesh):
    ctx = R.Context(0)
    P, F = MESHES[mesh]()
    g = R.SurfaceGraph(F, P, ctx)
    m = R.LearnedModel(seed=3, ctx=ctx)
    rng = np.random.default_rng(8)
    w = m.get_parameters()
    w = (w + 0.05 * rng.standard_normal(w.size)).astype(np.float32)
    m.set_parameters(w)
    r, y = rng.standard_normal(3 * len(P)), 0.1 * rng.standard_normal(3 * len(P))
    zt = y + 0.02 * rng.standard_normal(3 * len(P))
    rd, yd, zd = (torch.tensor(v).cuda() for v in (r, y, zt))
    out = torch.zeros_like(rd)
    torch.cuda.synchronize()
    m.apply_device(g, 1, rd.data_ptr(), yd.data_ptr(), out.data_ptr())
    loss = m.loss_and_gradient_device(g, rd.data_ptr(), yd.data_ptr(), zd.data_ptr())
    z_ref, loss_ref, grad_ref = reference(w, static_features(P, F), one_ring(F, len(P)), r, y, zt)
    assert np.linalg.norm(out.cpu().numpy() - z_ref) <= 1e-5 * np.linalg.norm(z_ref)
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    assert np.linalg.norm(m.get_gradient().astype(np.float64) - grad_ref) <= 1e-3 * np.linalg.norm(grad_ref)
