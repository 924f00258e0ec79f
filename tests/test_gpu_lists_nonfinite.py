"""Particles at non-finite positions in 3D scenes of 65,536 particles and more, whose
lists are built one particle per lane (k_lists_lane).  They land in cell 1 of x and
y (or of z) with MPS_ERR_CELL and neighbour nothing.  There they may lie out of
x's order, which the list passes search by, so rows close to that cell may be short;
every other row is that of the scene without them, also where it shares a warp
with them, no row gains an entry, and the orders stay permutations."""
import numpy as np
import pytest

import voxarmps_b200 as vm
from voxarmps_b200 import cases, config
from gpu_util import gpu_cfg

pytestmark = pytest.mark.gpu

L0 = 0.005
NAN, MINUS_NAN = np.array([0x7ff8000000000000, 0xfff8000000000000], np.uint64).view(np.float64)
SPAN = 4  # cells along x that a warp's particles may span


def _lists(cfg, case):
    s = vm.Solver(cfg, case)
    r = s.init()
    out = [s.lists(which) + (s.get("cell_" + sfx), s.get("perm_" + sfx))
           for which, sfx in ((0, "s"), (1, "l"))]
    s.close()
    return r, out


def _keys(off, nbr, n):
    return np.repeat(np.arange(n), np.diff(off)).astype(np.int64) * n + nbr


@pytest.fixture(scope="module")
def scene():
    case = cases.dam_break(3, L0, (30, 40, 28), (74, 52, 28))
    assert len(case["x"]) >= 65_536
    cfg = config.reference_defaults(L0, 3)
    cfg.update(re_s=2.1 * L0, re_l=4.0 * L0, dt=5e-5, gy=-9.81)
    cfg = gpu_cfg(config.with_box(cfg, case))
    r, whole = _lists(cfg, case)
    assert r == 0
    return cfg, case, whole


@pytest.mark.parametrize("axes, value", [
    ("x", MINUS_NAN), ("x", np.inf), ("y", NAN), ("z", -np.inf), ("xyz", MINUS_NAN),
    ("xyz", np.inf)])
def test_rows_of_the_others(scene, axes, value):
    cfg, case, whole = scene
    n = len(case["x"])
    fluid = np.flatnonzero(np.asarray(case["ptype"]) > 0)
    bad = fluid[np.linspace(0, len(fluid) - 1, 40).astype(int)]
    broken = {k: np.array(v) if k in ("x", "y", "z") else v for k, v in case.items()}
    for k in axes:
        broken[k][bad] = value
    r, got = _lists(cfg, broken)
    assert r & vm.MPS_ERR_CELL
    gone = np.zeros(n, bool)
    gone[bad] = True
    for (off, nbr, cell, _), (goff, gnbr, _, perm), re in zip(whole, got,
                                                              (cfg["re_s"], cfg["re_l"])):
        assert np.array_equal(np.sort(perm), np.arange(n))
        assert not np.diff(goff)[gone].any()
        nx, ny = (int((cfg[a + "max"] - cfg[a + "min"]) / re) + 1 for a in "xy")
        ix, iy = (cell - 1) % nx + 1, (cell - 1) // nx % ny + 1
        near = (ix <= 2 + SPAN) & (iy <= 2)
        assert near.mean() < 0.1
        owner = np.repeat(np.arange(n), np.diff(off))
        keep = ~gone[owner] & ~gone[nbr]
        far, gfar = keep & ~near[owner], ~near[np.repeat(np.arange(n), np.diff(goff))]
        rows, grows = _keys(off, nbr, n), _keys(goff, gnbr, n)
        assert np.array_equal(rows[far], grows[gfar])
        assert np.isin(grows[~gfar], rows[keep]).all()
