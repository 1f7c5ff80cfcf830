"""mpcmd_collide_static against numpy in FP64 at the coordinates where its
fixed-point cell arithmetic hands over to FP64: on shifted cell faces and one
rounding to either side of them, on cell faces, at 0 and the box edge, outside
a periodic box, and tiny offsets; both geometries and both senses, small and
uneven boxes.  A particle put into another cell changes its velocity by the
order of a thermal velocity; equal cells leave FP64 rounding, 1e-12.
"""
import math

import numpy as np
import pytest

import main_gb300
from main_gb300 import config, contract_u01

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def reference(pos, vel, box, walls, angle, sense, seed, step):
    s = [contract_u01(seed, 1, 0, 0, step, 0) - 0.5, contract_u01(seed, 1, 0, 0, step, 1) - 0.5,
         contract_u01(seed, 1, 0, 1, step, 0) - 0.5]
    cell, off = [], []
    for q in range(3):
        f = np.floor(pos[q])
        c, o = f.astype(np.int64), pos[q] - f
        if q < 2 or not walls:
            c %= box[q]
        else:
            o = np.where(c >= box[q], 1.0, np.where(c < 0, 0.0, o))
            c = np.clip(c, 0, box[q] - 1)
        cell.append(c)
        off.append(o)
    k = [(cell[q] + np.floor(off[q] + s[q]).astype(np.int64)) % box[q] for q in range(2)]
    if walls:
        kz = cell[2] + np.floor(off[2] + s[2] + 1.0 if s[2] < 0 else off[2] + s[2]).astype(np.int64)
    else:
        kz = (cell[2] + np.floor(off[2] + s[2]).astype(np.int64)) % box[2]
    key = k[0] + box[0] * (k[1] + box[1] * kz)
    n = box[0] * box[1] * (box[2] + walls)
    cnt = np.maximum(np.bincount(key, minlength=n), 1)
    cm = [np.bincount(key, weights=v, minlength=n) / cnt for v in vel]
    axis = np.zeros((n, 3))
    for c in np.unique(key):
        phi = 2 * math.pi * contract_u01(seed, 2, int(c), 0, step, 0)
        t = 2 * contract_u01(seed, 2, int(c), 0, step, 1) - 1
        axis[c] = (math.sqrt(1 - t * t) * math.cos(phi), math.sqrt(1 - t * t) * math.sin(phi), t)
    u = axis[key]
    m = np.stack([c[key] for c in cm], axis=1)
    d = np.stack(vel, axis=1) - m
    co, si = math.cos(angle), math.sin(angle) * sense
    return m + co * d + (1 - co) * (u * d).sum(axis=1, keepdims=True) * u + si * np.cross(u, d), s


@pytest.mark.parametrize("box", [(1, 1, 1), (5, 3, 7), (16, 16, 4), (80, 2, 3)])
@pytest.mark.parametrize("walls", [0, 1])
@pytest.mark.parametrize("sense", [1, -1])
def test_cells_at_faces(box, walls, sense):
    for step in (3, 4, 5, 6):                    # shifts of either sign
        n = 4001
        rng = np.random.default_rng(step)
        seed, angle = 11, 2.1
        vel = [rng.normal(size=n) for _ in range(3)]
        _, s = reference([np.zeros(1)] * 3, [np.zeros(1)] * 3, box, walls, angle, sense, seed, step)
        pos = []
        for q in range(3):
            L = box[q]
            face = rng.integers(0, L + 1, n).astype(np.float64)
            shifted = face - s[q]
            kind = rng.integers(0, 9, n)
            p = np.choose(kind, (rng.uniform(0, L, n), face, np.nextafter(face, -1.0), np.nextafter(face, L + 1.0),
                                 shifted, np.nextafter(shifted, -10.0), np.nextafter(shifted, 2000.0),
                                 rng.uniform(0, 1e-9, n), shifted + rng.uniform(-1e-9, 1e-9, n)))
            # a periodic box also takes coordinates outside it, walls take the clamped ones
            p += np.where(rng.random(n) < 0.1, rng.choice((-L, L), n), 0.0) if (q < 2 or not walls) else 0.0
            pos.append(p)
        ref, _ = reference(pos, vel, box, walls, angle, sense, seed, step)
        dp = [torch.as_tensor(p, device="cuda") for p in pos]
        dv = [torch.as_tensor(v, device="cuda") for v in vel]
        st = main_gb300.lib().mpcmd_collide_static(
            *[t.data_ptr() for t in dp + dv], n, *box, config.GEOM_WALLS if walls else config.GEOM_PERIODIC, angle,
            sense, seed, step, torch.cuda.current_stream().cuda_stream)
        assert st == 0
        got = np.stack([v.cpu().numpy() for v in dv], axis=1)
        assert np.abs(got - ref).max() <= 1e-12, (step, np.abs(got - ref).max())
