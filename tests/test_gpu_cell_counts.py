"""The particle counts of the shifted cells (mpcmd_get_cell_rotation): zeros before the
first rotation stage call, every particle after one, and their memory in boxes of
more than 2^22 cells taken only by a context that makes the call."""
import numpy as np
import pytest

from gpu_helpers import CASES
from main_gb300 import Engine, config

pytestmark = pytest.mark.gpu


def counted(cfg, grows):
    e = Engine(cfg)
    e.initial()
    before = e.device_bytes()
    assert not e.cell_rotation()[2].any() and e.device_bytes() == before
    for step in (50, 100):
        e.set_step(step)
        e.mpc_rotation()
        assert np.array_equal(e.cell_rotation()[2], np.bincount(e.new_cell(), minlength=e.n_cells_shifted()))
    assert e.device_bytes() == before + (4 * e.n_cells_shifted() if grows else 0)
    e.close()


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("case", ["c0", "c1"])
def test_small_boxes(case, prec):
    counted(CASES[case](prec), False)


@pytest.mark.parametrize("lx,lz,grows", [(256, 64, False), (257, 64, True), (256, 65, True)])
def test_large_boxes(lx, lz, grows):
    counted(config.base_config(lx=lx, ly=256, lz=lz, n_solvent=400001, seed=3, precision=32), grows)
