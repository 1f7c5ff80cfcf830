"""A training step (mpcmd_mlp_gradients, mpcmd_mlp_train_step) at the edges of
its row tiles (128, in pairs), widths, depths and output tiles (128 columns),
and with more row tiles than SMs.

Gradients: within 2e-2 relative L2 error of the FP64 gradient with BF16 at the
kernels' rounding points, the loss within 1e-3 (the bounds of the whole
network's test: a BF16 rounding that flips changes a value by 2^-8).  The first
Adam step from fresh moments: about a dozen FP32 operations without
cancellation on the gradient, so the update within 16 x 2^-24 of its FP64 value
and the parameter within one more rounding."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from main_gb300.surrogate import Mlp  # noqa: E402
from test_gpu_mlp import reference, relerr  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n_in,n_hidden,n_layers,n_out", [
    (128, 1, 64, 1, 1), (128, 8, 64, 2, 64), (256, 33, 128, 3, 65), (384, 64, 192, 1, 128), (384, 8, 192, 4, 129),
    (640, 8, 256, 16, 300), (256, 8, 256, 4, 2050), (128, 5, 64, 2, 4097), (39168, 3, 64, 3, 17)])
def test_step(batch, n_in, n_hidden, n_layers, n_out):
    lr, eps = 1e-3, 1e-8
    net = Mlp(n_in=n_in, n_hidden=n_hidden, n_layers=n_layers, n_out=n_out, batch=batch, max_rows=batch, seed=2, lr=lr,
              eps=eps)
    rng = np.random.default_rng(n_out)
    p = net.params() + rng.normal(0, 0.05, net.n_params).astype(np.float32)   # (biases too)
    net.set_params(p)
    x = rng.normal(size=(batch, n_in)).astype(np.float32)
    t = rng.normal(size=(batch, n_out)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, n_out).astype(np.float32)
    g, loss = net.gradients(x, t, w)
    _, loss_ref, ref = reference(net.unflatten(p.astype(np.float64)), x.astype(np.float64), t.astype(np.float64),
                                 w.astype(np.float64))
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    for l, ((gw, gb), (rw, rb)) in enumerate(zip(net.unflatten(g.astype(np.float64)), ref)):
        assert relerr(gw, rw) <= 2e-2 and relerr(gb, rb) <= 2e-2, l
    loss1 = net.train_step(*(torch.as_tensor(q, device="cuda") for q in (x, t, w)))
    assert loss1 == loss
    g64, b1, b2 = g.astype(np.float64), float(np.float32(0.9)), float(np.float32(0.999))
    m = float(np.float32(1) - np.float32(0.9)) * g64 / float(np.float32(1.0 - 0.9))
    v = float(np.float32(1) - np.float32(0.999)) * g64 * g64 / float(np.float32(1.0 - 0.999))
    up = float(np.float32(lr)) * m / (np.sqrt(v) + float(np.float32(eps)))
    want = p.astype(np.float64) - up
    bound = 2.0 ** -24 * np.abs(want) + 16 * 2.0 ** -24 * np.abs(up)
    assert (np.abs(net.params() - want) <= bound).all()
    net.close()
