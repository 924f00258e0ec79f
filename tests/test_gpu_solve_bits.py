"""An FP64 pressure solve gives the same bits in its two forms: in one cooperative
launch (k_cg_loop) and as one launch per kernel, which profiled steps take.  The
one launch forms the launches' own sums over the launches' own grid, so nothing of
it shows in a scene that magnifies a difference of rounding (Herschel-Bulkley
viscosity, which grows as 1 / sqrt(II) where the shear vanishes)."""
import numpy as np
import pytest

import voxarmps_b200 as vm
from voxarmps_b200 import cases, config
from gpu_util import gpu_cfg

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "u", "v", "w", "p")


def _dam(dim, fluid, tank, **kw):
    l0 = 0.01 if dim == 2 else 0.005
    case = cases.dam_break(dim, l0, fluid, tank)
    cfg = config.reference_defaults(l0, dim)
    cfg.update(re_s=2.1 * l0, re_l=4.0 * l0, dt=1e-4 if dim == 2 else 5e-5, gy=-9.81)
    return gpu_cfg(config.with_box(cfg, case), **kw), case


def _two_phase(w, h, **kw):
    """Column of a Herschel-Bulkley fluid in a Newtonian one, with SPS."""
    l0 = 0.002
    block = (cases.FLUID2, (0, h), (w // 4, h + h // 2))
    case = cases.dam_break(2, l0, (w, h), (w, 3 * h), blocks=[block])
    cfg = config.reference_defaults(l0, 2)
    cfg.update(re_s=2.1 * l0, re_l=4.0 * l0, gy=-9.81, dt=1e-4, turb=1, cs=0.12, rho2=900.0,
               nu2=1e-4, fluid2_type=1, n_pl=1.0, meu0=1e-4 * 900.0, cohes=5.0, phi=0.0)
    return gpu_cfg(config.with_box(cfg, case), **kw), case


def _flow(cfg, case, seed):
    """A flowing state: displaced fluid, a smooth velocity field with noise."""
    rng = np.random.default_rng(seed)
    dim, l0 = cfg["dim"], cfg["l0"]
    fl = np.asarray(case["ptype"]) > 0
    s = {k: np.array(case[k], np.float64) for k in FIELDS}
    ext = s["x"].max()
    for k in FIELDS[:dim]:
        s[k][fl] += rng.uniform(-0.04, 0.04, fl.sum()) * l0
    px, py = s["x"][fl] * np.pi / ext, s["y"][fl] * np.pi / ext
    s["u"][fl] = 0.1 * np.sin(px) * np.cos(py) + rng.normal(0, 0.01, fl.sum())
    s["v"][fl] = -0.1 * np.cos(px) * np.sin(py) + rng.normal(0, 0.01, fl.sum())
    s["p"][fl] = 9810 * (s["y"].max() - s["y"][fl]) * rng.uniform(0.95, 1.05, fl.sum())
    return s


def _ptrs(d, dim):
    return [d[k].ctypes.data if dim == 3 or k not in ("z", "w") else 0 for k in FIELDS]


def _run(cfg, case, profile, steps, tuning=None, learned=False, seed=5):
    s = vm.Solver(cfg, case)
    assert s.init() == 0
    if learned:
        s.gnn_create(4, 1)
        w = s.gnn_params()
        s.gnn_params(set_to=w + np.random.default_rng(3).normal(0, 0.02, w.size)
                     .astype(np.float32))
        s.gnn_use(True)
    if tuning is not None:
        s.set_tuning(s.get_tuning()["small_lanes"], tuning)
    s.set_profile(profile)
    state = _flow(cfg, case, seed)
    s.set_state(*_ptrs(state, cfg["dim"]))
    figures = []
    for _ in range(steps):
        s.step()
        assert s.scalar("one_launch_solve") == (0 if profile else 1)
        figures.append([s.scalar(k) for k in ("cg_iters", "cg_relres", "cg_r0")])
    out = {k: s.get(k) for k in FIELDS + ("pnew", "phat")}
    s.close()
    return out, np.array(figures)


def _same(cfg, case, steps=2, **kw):
    (a, fa), (b, fb) = (_run(cfg, case, profile, steps, **kw) for profile in (False, True))
    assert fa[:, 0].min() >= 1
    assert np.array_equal(fa.view(np.uint64), fb.view(np.uint64))
    for k in a:
        assert np.array_equal(a[k].view(np.uint64), b[k].view(np.uint64)), k


@pytest.mark.parametrize("dim, fluid, tank", [
    (2, (3, 5), (4, 6)),               # 93: one block, most rows walls
    (2, (20, 10), (24, 15)),           # 380
    (2, (16, 20), (18, 20)),           # 512: the last of one block
    (2, (15, 21), (18, 21)),           # 513: nine blocks
    (2, (25, 50), (100, 60)),          # 1,928
    (2, (100, 130), (842, 140)),       # 16,384: the last of the smaller grid
    (2, (100, 131), (809, 140)),       # 16,385
    (2, (151, 200), (430, 210)),       # 32,768: the last that forms p as it gathers
    (2, (150, 200), (497, 210)),       # 32,769
    (3, (4, 6, 3), (4, 6, 3)),         # 732, rows of one block's walls on all sides
    (3, (9, 11, 7), (30, 14, 9)),      # 6,093
    (3, (20, 40, 20), (80, 50, 20)),   # 54,508
    (3, (45, 74, 46), (82, 82, 46)),   # 232,836: several virtual blocks of vectors per quarter
    (2, (512, 500), (1002, 520)),      # 262,144: the last of one launch
])
def test_dam(dim, fluid, tank):
    _same(*_dam(dim, fluid, tank))


def test_one_row_more_takes_the_launches():
    cfg, case = _dam(2, (512, 502), (661, 520))
    assert len(case["x"]) == 262_145
    s = vm.Solver(cfg, case)
    assert s.init() == 0 and s.step() == 0
    assert s.scalar("one_launch_solve") == 0
    s.close()


@pytest.mark.parametrize("w, h", [(24, 16), (80, 40), (203, 61), (600, 100)])
def test_two_phase_shear_thinning(w, h):
    _same(*_two_phase(w, h), steps=4)


@pytest.mark.parametrize("opts", [dict(warm_start=0), dict(warm_start=2), dict(solver=2),
                                  dict(srcopt=1), dict(matopt=1), dict(cg_max=3)], ids=str)
def test_options(opts):
    _same(*_dam(2, (40, 60), (100, 70), **opts))


@pytest.mark.parametrize("blocks_per_sm", [1, 3, 5])
@pytest.mark.parametrize("fluid, tank", [((25, 50), (100, 60)), ((300, 300), (320, 310))])
def test_grids_of_the_tuning(blocks_per_sm, fluid, tank):
    _same(*_dam(2, fluid, tank), tuning=blocks_per_sm)


@pytest.mark.parametrize("fluid, tank", [((25, 50), (100, 60)), ((150, 150), (200, 160))])
def test_network_guess(fluid, tank):
    _same(*_dam(2, fluid, tank), learned=True)
