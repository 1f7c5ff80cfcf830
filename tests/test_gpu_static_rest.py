"""mpcmd_collide_static leaves a particle alone in its cell, and particles at rest
relative to one another, their velocities bit for bit: v - v_cm is zero there (the
sum of 1, 2 or 4 equal velocities and its mean are exact).  Sets that form their
cells' maps themselves (up to 8,192 particles), sets whose kernels start early and
larger ones; both geometries and senses; speeds of every magnitude."""
import numpy as np
import pytest

import main_gb300
from main_gb300 import config

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walls", [0, 1])
@pytest.mark.parametrize("sense", [1, -1])
@pytest.mark.parametrize("edge,copies", [(8, 1), (8, 4), (32, 2), (64, 1), (64, 4)])
def test_velocities_kept(edge, copies, walls, sense):
    rng = np.random.default_rng(edge + copies)
    site = np.stack(np.meshgrid(*[np.arange(0.25, edge, 2.0)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    site = site + rng.uniform(0, 0.9, site.shape)      # never two sites in one shifted cell
    v = rng.normal(size=site.shape) * 10.0 ** rng.uniform(-8, 8, site.shape)
    order = rng.permutation(len(site) * copies)
    pos, vel = np.repeat(site, copies, axis=0)[order], np.repeat(v, copies, axis=0)[order]
    dp = [torch.as_tensor(np.ascontiguousarray(pos[:, q]), device="cuda") for q in range(3)]
    dv = [torch.as_tensor(np.ascontiguousarray(vel[:, q]), device="cuda") for q in range(3)]
    for step in range(4):
        st = main_gb300.lib().mpcmd_collide_static(
            *[t.data_ptr() for t in dp + dv], len(pos), edge, edge, edge,
            config.GEOM_WALLS if walls else config.GEOM_PERIODIC, 2.1, sense, 11, step,
            torch.cuda.current_stream().cuda_stream)
        assert st == 0
    for q in range(3):
        assert np.array_equal(dv[q].cpu().numpy(), vel[:, q])
