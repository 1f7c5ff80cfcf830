"""Inference (mpcmd_mlp_forward) at the edges of its row tiles (128), output
tiles (256 columns, the last one narrower), widths and depths, and of the
split of row tiles over the SMs: outputs within 1e-2 of their scale of the
FP64 network with BF16 at the kernel's rounding points, and every row
bit-identical whatever call it is part of (a row's arithmetic does not depend
on its tile, on how the output tiles are split, or on the other rows)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from main_gb300.surrogate import Mlp  # noqa: E402
from test_gpu_mlp import reference  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_hidden,n_layers,n_out", [
    (1, 64, 1, 1), (8, 64, 3, 16), (33, 128, 2, 17), (64, 192, 4, 255), (8, 256, 1, 256), (8, 256, 4, 257),
    (8, 256, 16, 300), (8, 256, 4, 2050), (5, 192, 2, 4097)])
def test_shapes(n_in, n_hidden, n_layers, n_out):
    net = Mlp(n_in=n_in, n_hidden=n_hidden, n_layers=n_layers, n_out=n_out, batch=128, max_rows=1000, seed=2)
    p = net.params()
    p += np.random.default_rng(0).normal(0, 0.05, p.size).astype(np.float32)   # (biases too)
    net.set_params(p)
    rng = np.random.default_rng(1)
    x = rng.normal(size=(1000, n_in)).astype(np.float32)
    y = net.forward(x).cpu().numpy()
    ref = reference(net.unflatten(p.astype(np.float64)), x.astype(np.float64))
    assert np.abs(y - ref).max() <= 1e-2 * np.abs(ref).max()
    for rows in (1, 31, 127, 128, 129, 257):
        assert np.array_equal(net.forward(x[:rows]).cpu().numpy(), y[:rows]), rows
    net.close()


def test_waves():
    # 152 SMs: full rounds, one row tile more, and left-overs that split two ways and not at all
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    net = Mlp(n_out=300, batch=128, max_rows=(2 * sms + 9) * 128, seed=4)
    rng = np.random.default_rng(3)
    x = torch.as_tensor(rng.normal(size=((2 * sms + 9) * 128, 8)).astype(np.float32), device="cuda")
    whole = torch.cat([net.forward(x[i:i + 1024]) for i in range(0, len(x), 1024)])
    for tiles, ragged in ((sms, 0), (sms, 1), (sms - 1, 77), (2 * sms, 1), (2 * sms + 8, 5), (sms // 2, 3), (sms // 2 + 1, 0)):
        rows = tiles * 128 + ragged
        assert torch.equal(net.forward(x[:rows]), whole[:rows]), (tiles, ragged)
    net.close()
