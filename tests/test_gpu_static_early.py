"""mpcmd_collide_static where its kernels start while the one before them ends
(up to three blocks of 256 particles an SM), at that edge and at the edge of the
sets that form their own cells' maps (8,192): three collisions issued back to
back, and the same as a captured graph replayed, against numpy in FP64.  One
collision leaves FP64 rounding, 1e-12; three leave three times that."""
import numpy as np
import pytest

import main_gb300
from main_gb300 import config
from test_gpu_static_rotate import reference

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BOX, ANGLE, SEED = (12, 10, 9), 2.1, 11


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("size", ["1", "255", "8192", "8193", "edge", "edge+1"])
def test_chained_collisions(size, captured):
    edge = 3 * 256 * torch.cuda.get_device_properties(0).multi_processor_count
    n = edge + size.count("+") if size.startswith("edge") else int(size)
    rng = np.random.default_rng(n)
    pos = [rng.uniform(0, L, n) for L in BOX]
    vel = [rng.normal(size=n) for _ in range(3)]
    dp = [torch.as_tensor(p, device="cuda") for p in pos]

    def collide(dv, steps):
        for step in steps:
            st = main_gb300.lib().mpcmd_collide_static(
                *[t.data_ptr() for t in dp + dv], n, *BOX, config.GEOM_PERIODIC, ANGLE, 1, SEED, step,
                torch.cuda.current_stream().cuda_stream)
            assert st == 0

    dv = [torch.as_tensor(v, device="cuda") for v in vel]
    if captured:
        collide([v.clone() for v in dv], (1,))   # (sets the device up outside the capture)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            collide(dv, (3, 4, 5))
        graph.replay()
    else:
        collide(dv, (3, 4, 5))
    torch.cuda.synchronize()
    ref = vel
    for step in (3, 4, 5):
        ref = list(reference(pos, ref, BOX, 0, ANGLE, 1, SEED, step)[0].T)
    got = np.stack([v.cpu().numpy() for v in dv])
    assert np.abs(got - np.stack(ref)).max() <= 3e-12
