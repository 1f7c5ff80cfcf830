"""Training batches of several row tiles a CTA: the backward chain then takes the
next input as soon as its last layer is done, with no output job between them
(one and two layers of the chain, up to five rounds and a part of one).

Gradients and loss within the bounds of the single steps (2e-2 relative L2 and
1e-3), repeated passes bit for bit the same (no sum of theirs depends on order)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from main_gb300.surrogate import Mlp  # noqa: E402
from test_gpu_mlp import reference, relerr  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_layers,rounds,more", [(2, 1, 1), (2, 5, 3), (3, 2, 0)])
def test_rounds(n_layers, rounds, more):
    batch = 128 * (rounds * torch.cuda.get_device_properties(0).multi_processor_count + more)
    net = Mlp(n_in=3, n_hidden=64, n_layers=n_layers, n_out=5, batch=batch, max_rows=batch, seed=2)
    rng = np.random.default_rng(rounds)
    p = net.params()
    x = rng.normal(size=(batch, 3)).astype(np.float32)
    t = rng.normal(size=(batch, 5)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, 5).astype(np.float32)
    g, loss = net.gradients(x, t, w)
    _, loss_ref, ref = reference(net.unflatten(p.astype(np.float64)), x.astype(np.float64), t.astype(np.float64),
                                 w.astype(np.float64))
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    for l, ((gw, gb), (rw, rb)) in enumerate(zip(net.unflatten(g.astype(np.float64)), ref)):
        assert relerr(gw, rw) <= 2e-2 and relerr(gb, rb) <= 2e-2, l
    for _ in range(20):
        g2, loss2 = net.gradients(x, t, w)
        assert loss2 == loss and np.array_equal(g2, g)
    net.close()
