"""The system series (mpcmd_observables, mpcmd_ens_observables) against numpy
sums of the downloaded state, at particle counts around the kernels' groups
of four particles and the ensemble's work tiles.

Bounds: sums of N terms rounded to 2^-24 each would leave about 2^-24 sqrt(N)
of one term's size (the engine may leave 10 times that); the ensemble's sums
are exact products added with 2^-45 relative error, so they match the FP64
sums of the same numbers to 1e-12 of the sum of magnitudes.  Species counts
are exact.
"""
import numpy as np
import pytest

from main_gb300 import Engine, config, ensemble

pytestmark = pytest.mark.gpu

MASSES = [(1.0, 1.7, 0.3, 2.0 / 3.0), (2.0 / 3.0,) * 4]


def sums(st, mass):
    m = np.asarray(mass)[st["flag"]]
    v = [st[k] for k in ("vx", "vy", "vz")]
    mom = np.array([(m * c).sum() for c in v])
    scale = np.array([(m * np.abs(c)).sum() for c in v])
    kin = 0.5 * (m * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)).sum()
    return mom, scale, kin, np.bincount(st["flag"], minlength=4)


@pytest.mark.parametrize("mass", MASSES)
@pytest.mark.parametrize("extra", [0, 1, 2, 3, 511])
def test_engine_series(extra, mass):
    n = 10 * 16 ** 3 + extra
    cfg = config.base_config(lx=16, ly=16, lz=16, n_solvent=n, mass=list(mass), precision=32, seed=3)
    e = Engine(cfg)
    e.initial()
    st = e.download_state()
    st["flag"] = np.random.default_rng(extra).integers(0, 4, n).astype(np.int32)
    e.upload_state(st)
    e.prepare()
    e.run(7)                      # some states live in the shell buffer
    o = e.observables()
    mom, scale, kin, cnt = sums(e.download_state(), mass)
    term = scale.max() / n
    assert np.abs(o["solvent_momentum"] - mom).max() <= 10 * 2.0 ** -24 * np.sqrt(n) * term
    assert abs(o["kinetic_solvent"] - kin) <= 10 * 2.0 ** -24 / np.sqrt(n) * kin
    assert np.array_equal(o["species_count"], cnt)


@pytest.mark.parametrize("mass", MASSES)
@pytest.mark.parametrize("schedule", [(64, 32, 32), (1000, 96, 64), (4096, 256, 128)])
def test_ensemble_series(schedule, mass):
    reps = [ensemble.replica(16, n_solvent=n, seed=5 + n, rc=2.0, rn=1.0, dcn=3.6, mass=mass)
            for n in (4095, 4096, 4097, 20483)]
    ens = ensemble.Ensemble(reps, precision=32, schedule=schedule)
    ens.initial()
    ens.prepare()
    rng = np.random.default_rng(1)
    for r, rep in enumerate(reps):
        st = ens.download(r)
        st["flag"] = rng.integers(0, 4, rep["n_solvent"]).astype(np.int32)
        ens.upload(r, st)
    obs = ens.observables()
    for r in range(len(reps)):
        mom, scale, kin, cnt = sums(ens.download(r), mass)
        assert np.all(np.abs(obs[r]["solvent_momentum"] - mom) <= 1e-12 * scale)
        assert abs(obs[r]["kinetic_solvent"] - kin) <= 1e-12 * kin
        assert np.array_equal(obs[r]["species_count"], cnt)
