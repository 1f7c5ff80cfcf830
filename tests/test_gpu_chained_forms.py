"""The chained kernels of test_gpu_chained_steps in their other forms: the FP32
build (its own pair-force sums, RATTLE and block sizes), rotors, owner tags, and
boxes whose particles an order-only re-sort has moved, with dimer counts on either
side of the eight blocks of eight up to which the dimer kernel is chained.  One
call of 55 steps against 55 calls of one step.

FP64: 1e-9, as there.  FP32: the bounds of the FP32 trajectories against the
oracle over a hundred steps, 2e-4 in position and 2e-3 in velocity (a state read
one step too early is off by a flight of one step, 5e-3 to 1e-2)."""
import numpy as np
import pytest

from gpu_helpers import assert_close
from main_gb300 import Engine, config

pytestmark = pytest.mark.gpu

ROTORS_81 = dict(n_dimers=81, layout_rows=9, layout_cols=9, lx=128, ly=128, lz=16)
FORMS = {
    "dimers_8": ("c1", dict(scale=0.5, n_dimers=8), 0),
    "dimers_64": ("c1", dict(n_dimers=64), 0),
    "dimers_65": ("c1", dict(n_dimers=65), 0),
    "resorted_64": ("c1", dict(n_dimers=64), 1),
    "resorted_65": ("c1", dict(n_dimers=65), 1),
    "rotors_9": ("rot", dict(scale=0.5), 0),
    "rotors_81": ("rot", ROTORS_81, 0),
    "rotors_81_resorted": ("rot", ROTORS_81, 1),
    "owner": ("rot_owner", dict(scale=0.25, sort_every=40, k=[0.5, 0, 0, 0, 0, 0]), 0),
    "owner_resorted": ("rot_owner", dict(scale=0.25, k=[0.5, 0, 0, 0, 0, 0]), 1),
}


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("form", list(FORMS))
def test_one_call_equals_single_steps(form, precision):
    name, kw, resort = FORMS[form]
    cfg = config.workload(name, seed=3, precision=precision, **kw)
    states, owners = [], []
    for chunk in (55, 1):
        e = Engine(cfg)
        e.initial()
        if resort:
            e.set_resort(cfg["mpc_every"])
        e.prepare()
        for _ in range(0, 55, chunk):
            e.run(chunk)
        assert (e.counters()["resorts"] > 0) == bool(resort)
        states.append(e.download_state())
        owners.append(e.get_owner_tags() if cfg["owner_tags"] else np.zeros(1))
        e.close()
    if precision == 64:
        assert_close(states[0], states[1], cfg, pos=1e-9, vel=1e-9, flags=1.0, dimer=1e-9)
        assert np.array_equal(owners[0], owners[1])
    else:
        assert_close(states[0], states[1], cfg, pos=2e-4, vel=2e-3, flags=0.999, dimer=2e-4)
        assert (owners[0] == owners[1]).mean() >= 0.999
