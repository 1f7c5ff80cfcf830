"""The system series of an FP32 ensemble keep the bits of FP64 sums.

Velocities chosen so that sums that keep fewer lose them: a few large ones among
many small ones that use all 24 bits (every thread of a block meets the same
pattern, so its rounding errors do not average out), and speeds whose squares
leave FP32's exponents.  Expected: exactly rounded sums of the same numbers.
Bound: an FP64 sum along the kernel's chain of additions (16 particles a thread, a
warp, 8 warps, one or two blocks) rounds at most 32 times, each by 2^-53 of the sum of
magnitudes; products with the masses two times more."""
import math

import numpy as np
import pytest

from main_gb300 import ensemble

pytestmark = pytest.mark.gpu

N = 4096
ONE, FOUR = (1.0 / 3.0,) * 4, (1.0, 1.7, 0.3, 2.0 / 3.0)


def velocities(kind):
    rng = np.random.default_rng(1)
    if kind == "mixed":
        v = np.repeat([[57.01413], [-57.130342], [56.933136]], N, axis=1)
        v[:, :256] = [[2.0 ** 30], [-2.0 ** 30], [2.0 ** 30]]
    elif kind == "huge":
        v = rng.normal(size=(3, N)) * 1e25
    elif kind == "tiny":
        v = rng.normal(size=(3, N)) * 1e-25
    else:   # every magnitude, zeros among them
        v = rng.normal(size=(3, N)) * 10.0 ** rng.uniform(-30, 30, (3, N))
        v[0, ::7] = 0.0
    return v.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("mass", [ONE, FOUR], ids=["one_mass", "four_masses"])
@pytest.mark.parametrize("kind", ["mixed", "huge", "tiny", "spread"])
def test_fp64_sums(kind, mass):
    rep = ensemble.replica(16, n_solvent=N, seed=5, rc=2.0, rn=1.0, dcn=3.6, mass=mass)
    ens = ensemble.Ensemble([rep], precision=32, schedule=(N, 256, 256))
    ens.initial()
    st = ens.download(0)
    st["vx"], st["vy"], st["vz"] = velocities(kind)
    st["flag"] = (np.arange(N) % 4).astype(np.int32)
    ens.upload(0, st)
    got = ens.download(0)
    assert np.array_equal(got["vx"], st["vx"]) and np.array_equal(got["flag"], st["flag"])
    o = ens.observables()[0]
    m = np.asarray(mass)[st["flag"]]
    for q, k in enumerate(("vx", "vy", "vz")):
        t = m * st[k]
        assert abs(o["solvent_momentum"][q] - math.fsum(t)) <= 34 * 2.0 ** -53 * math.fsum(np.abs(t)), k
    kin = math.fsum(np.concatenate([0.5 * m * st[k] ** 2 for k in ("vx", "vy", "vz")]))
    assert abs(o["kinetic_solvent"] - kin) <= 34 * 2.0 ** -53 * kin
    ens.close()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_not_finite(bad):
    rep = ensemble.replica(16, n_solvent=N, seed=5, rc=2.0, rn=1.0, dcn=3.6, mass=ONE)
    ens = ensemble.Ensemble([rep], precision=32)
    ens.initial()
    st = ens.download(0)
    st["vy"][77] = bad
    ens.upload(0, st)
    o = ens.observables()[0]
    assert np.isfinite(o["solvent_momentum"][[0, 2]]).all()
    assert np.array_equal(o["solvent_momentum"][1], bad, equal_nan=True)
    assert np.array_equal(o["kinetic_solvent"], abs(bad), equal_nan=True)
    ens.close()
