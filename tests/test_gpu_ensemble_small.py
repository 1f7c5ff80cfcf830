"""Replica counts around the one block of 32 replicas that takes the dimer step
of small ensembles, and hundreds of replicas of a few hundred particles: a block's share of a
rebuild (units of 256 particles) and of the observables (neighbouring work
tiles) then begins and ends inside replicas and covers several of them.

FP64: replicas of 255, 256, 257 and 40 particles follow their single-context
runs to the bounds of the larger ensembles (1e-9).  FP32: every replica's
series matches the FP64 sums of its downloaded state to 1e-12 of the sum of
magnitudes (the sums' relative error is 2^-45), the counts exactly."""
import numpy as np
import pytest

from gpu_helpers import assert_close
from main_gb300 import Engine
from main_gb300 import ensemble as E
from test_gpu_observables import sums

pytestmark = pytest.mark.gpu

SIZES = (255, 256, 257, 40, 513)


def replicas(count):
    return [E.replica(16, n_solvent=SIZES[i % len(SIZES)], seed=90 + i, rc=2.0, rn=1.0, dcn=3.6) for i in range(count)]


def test_fp64_follows_single_contexts():
    reps = replicas(700)
    picked = (0, 1, 2, 3, 352, 697, 699)
    ens = E.Ensemble(reps, precision=64)
    ens.initial()
    engines = {}
    for r in picked:
        cfg = E.config_of_replica(reps[r], precision=64)
        e = Engine(cfg)
        e.initial()
        ens.upload(r, e.download_state())
        e.prepare()
        engines[r] = (cfg, e)
    ens.prepare()
    for chunk in (50, 20):
        ens.run(chunk)
        for r, (cfg, e) in engines.items():
            e.run(chunk)
            assert_close(ens.download(r), e.download_state(), cfg, pos=1e-9, vel=1e-9, flags=1.0, dimer=1e-9)
    ens.close()


@pytest.mark.parametrize("count", [1, 7, 8, 31, 32, 33])
def test_fp64_dimer_blocks(count):
    reps = replicas(count)
    ens = E.Ensemble(reps, precision=64)
    ens.initial()
    engines = []
    for r in sorted({0, count // 2, count - 1}):
        cfg = E.config_of_replica(reps[r], precision=64)
        e = Engine(cfg)
        e.initial()
        ens.upload(r, e.download_state())
        e.prepare()
        engines.append((r, cfg, e))
    ens.prepare()
    for chunk in (50, 20, 3):
        ens.run(chunk)
        for r, cfg, e in engines:
            e.run(chunk)
            assert_close(ens.download(r), e.download_state(), cfg, pos=1e-9, vel=1e-9, flags=1.0, dimer=1e-9)
    ens.close()


@pytest.mark.parametrize("schedule", [(0, 0, 0), (64, 32, 32), (1000, 96, 64)])
def test_fp32_series(schedule):
    reps = replicas(300)
    ens = E.Ensemble(reps, precision=32, schedule=schedule)
    ens.initial()
    ens.prepare()
    ens.run(60)
    obs = ens.observables()
    for r, rep in enumerate(reps):
        mom, scale, kin, cnt = sums(ens.download(r), rep["mass"])
        assert np.all(np.abs(obs[r]["solvent_momentum"] - mom) <= 1e-12 * scale), r
        assert abs(obs[r]["kinetic_solvent"] - kin) <= 1e-12 * kin, r
        assert np.array_equal(obs[r]["species_count"], cnt), r
    ens.close()
