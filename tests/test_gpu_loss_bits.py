"""The training loss keeps the bits of an FP64 sum of its FP32 terms w (y - t)^2.

A network of zero parameters puts out zeros, so the terms are fl(fl(w t) t)
exactly: a large one among many small ones that use all 24 bits (the same in every
row, so that rounding errors do not average out), sums beyond FP32's largest
number, and terms that are no numbers.  Bound: the chunks of a row tile, a warp
and the partial sums are added in FP64, fewer than 64 roundings of 2^-53 each."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from main_gb300.surrogate import Mlp  # noqa: E402

pytestmark = pytest.mark.gpu


def loss_of(w, t, batch):
    net = Mlp(n_in=2, n_hidden=64, n_layers=1, n_out=len(t), batch=batch, max_rows=batch, seed=2)
    net.set_params(np.zeros(net.n_params, np.float32))
    x = np.zeros((batch, 2), np.float32)
    _, loss = net.gradients(x, np.tile(t, (batch, 1)), w)
    net.close()
    return loss


@pytest.mark.parametrize("batch", [128, 384])
@pytest.mark.parametrize("n_out", [32, 300])
def test_small_terms_beside_large_ones(n_out, batch):
    w, t = np.full(n_out, 57.01413, np.float32), np.ones(n_out, np.float32)
    w[::32], t[::32] = 1.0, 2.0 ** 15
    want = math.fsum((w * t * t).astype(np.float64))
    assert abs(loss_of(w, t, batch) - want) <= 64 * 2.0 ** -53 * want


def test_terms_below_the_normal_numbers():
    w, t = np.full(40, 1e-20, np.float32), np.full(40, 3e-10, np.float32)
    want = math.fsum((w * t * t).astype(np.float64))
    assert 0 < want < 1e-37 and abs(loss_of(w, t, 128) - want) <= 64 * 2.0 ** -53 * want


def test_sum_beyond_fp32():
    w, t = np.full(200, 0.7, np.float32), np.linspace(1e19, 2e19, 200).astype(np.float32)
    term = w * t * t
    assert np.isfinite(term).all()
    want = math.fsum(term.astype(np.float64))
    assert want > 3.5e38 and abs(loss_of(w, t, 256) - want) <= 64 * 2.0 ** -53 * want


@pytest.mark.parametrize("bad,loss", [(1e25, np.inf), (np.inf, np.inf), (np.nan, np.nan)])
def test_terms_that_are_no_numbers(bad, loss):
    w, t = np.ones(70, np.float32), np.ones(70, np.float32)
    t[41] = bad
    assert np.array_equal(loss_of(w, t, 128), loss, equal_nan=True)
