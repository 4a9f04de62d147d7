"""The learned correction's ring means where their lanes change: one channel a thread when the longest ring is above 64
and above a 128th of the vertices, else four. Against the plain PyTorch reference, within the tolerances of
test_learned_gpu."""
import numpy as np
import pytest

import rs_gb300 as R
from test_learned_gpu import one_ring, reference, static_features

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def fans(m, k):
    """m disks, 3 apart: a hub and k rim vertices that alternate in height."""
    a = 2.0 * np.pi * np.arange(k) / k
    one = np.vstack([np.zeros((1, 3)), np.c_[np.cos(a), np.sin(a), 0.3 * np.cos(5 * a)]])
    i = np.arange(k)
    face = np.c_[0 * i, 1 + i, 1 + (i + 1) % k]
    P = np.concatenate([one + [3.0 * (s % 12), 3.0 * (s // 12), 0.0] for s in range(m)])
    return P, np.concatenate([face + s * (k + 1) for s in range(m)]).astype(np.uint32)


# rings of 64 and 65 on few vertices, of 65 at 128 vertices a neighbour and just below
@pytest.mark.parametrize("m,k", [(3, 64), (3, 65), (126, 65), (127, 65), (2, 500)])
def test_forward_and_gradient(m, k):
    ctx = R.Context(0)
    P, F = fans(m, k)
    g = R.SurfaceGraph(F, P, ctx)
    model = R.LearnedModel(seed=3, ctx=ctx)
    rng = np.random.default_rng(8)
    w = model.get_parameters()
    w = (w + 0.05 * rng.standard_normal(w.size)).astype(np.float32)
    model.set_parameters(w)
    r, y = rng.standard_normal(3 * len(P)), 0.1 * rng.standard_normal(3 * len(P))
    zt = y + 0.02 * rng.standard_normal(3 * len(P))
    rd, yd, zd = (torch.tensor(v).cuda() for v in (r, y, zt))
    out = torch.zeros_like(rd)
    torch.cuda.synchronize()
    model.apply_device(g, 1, rd.data_ptr(), yd.data_ptr(), out.data_ptr())
    loss = model.loss_and_gradient_device(g, rd.data_ptr(), yd.data_ptr(), zd.data_ptr())
    z_ref, loss_ref, grad_ref = reference(w, static_features(P, F), one_ring(F, len(P)), r, y, zt)
    assert np.linalg.norm(out.cpu().numpy() - z_ref) <= 1e-5 * np.linalg.norm(z_ref)
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    assert np.linalg.norm(model.get_gradient().astype(np.float64) - grad_ref) <= 1e-3 * np.linalg.norm(grad_ref)
