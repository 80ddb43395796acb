"""Weight gradients where a brick's (tap, channel) pairs are dealt out over
several CTAs or none, and bricks end beyond the grid: against the numpy oracle,
with test_learned_gpu.py's bounds (3e-2 of each layer's norm, cosine 0.999)."""
import numpy as np
import pytest

import oracle.nn_oracle as NO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (24, 40, 56), (40, 72, 64)])
def test_gradients(gpu_lib, shape):
    from importlib import import_module
    learned = import_module(gpu_lib.__name__ + ".learned")
    D, H, W = shape
    net = learned.Net(W, H, D, seed=21)
    p = net.params.copy()
    p += (np.random.default_rng(22).standard_normal(p.size) * 0.02).astype(np.float32)
    net.params = p
    r = np.random.default_rng(23)
    x = r.standard_normal(shape + (NO.CIN,)).astype(np.float32)
    t = r.standard_normal(shape).astype(np.float32) * 0.1
    loss, g = net.loss_grad(x, t)
    loss_ref, g_ref, _ = NO.loss_and_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - loss_ref) <= 1e-2 * loss_ref
    off = 0
    for l, (ci, co, _) in enumerate(NO.LAYERS):
        n = 27 * ci * co + co
        a, b = g[off:off + n].astype(np.float64), g_ref[off:off + n]
        off += n
        err = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
        cos = float(a @ b / max(np.linalg.norm(a) * np.linalg.norm(b), 1e-30))
        assert err < 3e-2 and cos > 0.999, (l, err, cos)
