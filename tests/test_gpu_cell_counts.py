"""The particle counts of the shifted cells (mpcmd_get_cell_rotation): zeros before the
first rotation stage call, every particle after one, and their memory taken only
by a context that makes the call."""
import numpy as np
import pytest

from gpu_helpers import CASES
from main_gb300 import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("case", ["c0", "c1"])
def test_counts(case, prec):
    e = Engine(CASES[case](prec))
    e.initial()
    e.prepare()
    e.run(3)
    before = e.device_bytes()
    assert not e.cell_rotation()[2].any() and e.device_bytes() == before
    e2 = Engine(CASES[case](prec))
    e2.initial()
    for step in (50, 100):
        e2.set_step(step)
        e2.mpc_rotation()
        assert np.array_equal(e2.cell_rotation()[2], np.bincount(e2.new_cell(), minlength=e2.n_cells_shifted()))
    assert e2.device_bytes() == before + 4 * e2.n_cells_shifted()
    e.close()
    e2.close()
