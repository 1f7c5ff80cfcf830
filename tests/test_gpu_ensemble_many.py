"""Thousands of small replicas: the block that ends a rebuild takes several rounds of
replicas, the dimer step changes its block size (above 2,048 replicas), and most MD
steps rebuild some replica.  FP64 replicas follow their single-context runs to the
bounds of the smaller ensembles (1e-9)."""
import pytest

from gpu_helpers import assert_close
from main_gb300 import Engine
from main_gb300 import ensemble as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [(0, 0, 0), (64, 32, 32), (1000, 96, 64)])
@pytest.mark.parametrize("count", [257, 2048, 2049])
def test_follows_single_contexts(count, schedule):
    sizes = (255, 40, 513, 1500)
    reps = [E.replica(16, n_solvent=sizes[i % 4], seed=90 + i, rc=2.0, rn=1.0, dcn=3.6) for i in range(count)]
    ens = E.Ensemble(reps, precision=64, schedule=schedule)
    ens.initial()
    engines = []
    for r in (0, 31, 32, 255, 256, count // 2 + 1, count - 1):
        cfg = E.config_of_replica(reps[r], precision=64)
        e = Engine(cfg)
        e.initial()
        ens.upload(r, e.download_state())
        e.prepare()
        engines.append((r, cfg, e))
    ens.prepare()
    for chunk in (50, 23):
        ens.run(chunk)
        for r, cfg, e in engines:
            e.run(chunk)
            assert_close(ens.download(r), e.download_state(), cfg, pos=1e-9, vel=1e-9, flags=1.0, dimer=1e-9)
    ens.close()
