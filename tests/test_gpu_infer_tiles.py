"""Inference at the edges of its 128-column output tiles: one tile not full, full, and
a second one whose MMA is 16 columns wide; with few rows, where every output tile
goes to a CTA of its own.  Outputs within 1e-2 of their scale of the FP64 network
with BF16 at the kernel's rounding points, and every row bit-identical whatever
call it is part of."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from main_gb300.surrogate import Mlp  # noqa: E402
from test_gpu_mlp import reference  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_out", [112, 113, 127, 128, 129, 144, 145, 384, 385])
def test_tiles(n_out):
    net = Mlp(n_in=8, n_hidden=128, n_layers=2, n_out=n_out, batch=128, max_rows=20000, seed=2)
    p = net.params()
    p += np.random.default_rng(0).normal(0, 0.05, p.size).astype(np.float32)   # (biases too)
    net.set_params(p)
    x = np.random.default_rng(1).normal(size=(20000, 8)).astype(np.float32)
    y = net.forward(x).cpu().numpy()
    ref = reference(net.unflatten(p.astype(np.float64)), x.astype(np.float64))
    assert np.abs(y - ref).max() <= 1e-2 * np.abs(ref).max()
    for rows in (1, 33, 128, 129, 300):
        assert np.array_equal(net.forward(x[:rows]).cpu().numpy(), y[:rows]), rows
    net.close()
