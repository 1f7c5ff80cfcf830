"""mpcmd_concentration where its FP32 arithmetic could decide a bin or a slab
differently from FP64: coordinates on bin faces and slab bounds and one
rounding away from them, widths that are no binary fractions, particle counts
around the groups of four, lagging states.  Bit-identical fields: the
oracle's binning of the downloaded state (whole counts over the same volumes).
"""
import numpy as np
import pytest

from main_gb300 import Engine, config
from oracle import oracle as O

pytestmark = pytest.mark.gpu

WIDTHS = [(0.5, 0.5, 0.5), (0.3, 0.7, 1.9), (1.0 / 3.0, 0.1, 16.0), (1.0, 2.0, 0.0625)]


def check(e, cfg, prm):
    got = e.concentration(*prm)
    st = e.download_state()
    ref = O.concentration(st["x"], st["y"], st["z"], st["flag"], (cfg["lx"], cfg["ly"], cfg["lz"]), prm)
    for k, v in ref.items():
        np.testing.assert_array_equal(got[k], v, err_msg=str((k, prm)))
    assert got["xy_a"].any() and got["yz_b"].any()


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("extra", [0, 1, 2, 3])
@pytest.mark.parametrize("widths", WIDTHS)
def test_faces_and_bounds(prec, extra, widths):
    L = 16
    n = 8000 + extra
    cfg = config.base_config(lx=L, ly=L, lz=L, n_solvent=n, precision=prec, n_dimers=0)
    rng = np.random.default_rng(extra)
    slab, hw = (7.3, 8.2, 8.1), 2.7
    st = {}
    for k, w, s in zip("xyz", widths, slab):
        p = rng.uniform(0.0, L, n)
        face = np.rint(p / w) * w                     # on a bin face, or a rounding off it
        near = np.nextafter(np.float32(face), np.float32(rng.choice((0.0, L), n))).astype(np.float64)
        bound = rng.choice((s - hw, s + hw), n)
        pick = rng.integers(0, 4, n)
        st[k] = np.clip(np.choose(pick, (p, face, near, bound)), 0.0, np.nextafter(np.float32(L), np.float32(0)))
    for k in ("vx", "vy", "vz"):
        st[k] = rng.normal(size=n)
    st["flag"] = rng.integers(0, 4, n).astype(np.int32)
    e = Engine(cfg)
    e.upload_state(st)
    e.prepare()
    check(e, cfg, slab + (hw,) + widths)


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("name,scale", [("c0", 0.55), ("c1", 0.25)])
def test_lagging_states(prec, name, scale):
    cfg = config.workload(name, scale=scale, precision=prec)
    e = Engine(cfg)
    e.initial()
    st = e.download_state()
    st["flag"][::3] = 1
    e.upload_state(st)
    e.prepare()
    e.run(50 + 37)                # between rebuilds: deferred and free-flight states lag
    check(e, cfg, (cfg["lx"] / 2, cfg["ly"] / 2, cfg["lz"] / 2, cfg["rc"] * 2 ** (1 / 6), 0.3, 0.5, 0.7))
