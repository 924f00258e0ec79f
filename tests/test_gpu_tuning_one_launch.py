"""The autotuner searches the CG grid only where the solve takes more than one launch:
elsewhere its steps would time nothing, and the value keeps what it was (8, as
many as fit, when it was unset)."""
import pytest

import voxarmps_b200 as vm
from voxarmps_b200 import cases, config
from gpu_util import gpu_cfg

pytestmark = pytest.mark.gpu

STEPS = 2
LANES, GRIDS = 2, 4  # candidates of each parameter


def _dam(**kw):
    cfg, case = config.baseline(0)
    return gpu_cfg(cfg, **kw), case, None


def _batch(**kw):
    l0 = 0.01
    scenes = [cases.dam_break(2, l0, (w, h), (100, 60)) for w, h in ((10, 20), (25, 50))]
    base = config.reference_defaults(l0, 2)
    base.update(re_s=2.1 * l0, re_l=4.0 * l0, dt=1e-4, gy=-9.81)
    cfg, case, sid, boxes, pmax = config.batched(gpu_cfg(base, **kw), scenes)
    return cfg, case, (sid, boxes, pmax)


MAKE = {"dam": _dam, "batch": _batch}


@pytest.mark.parametrize("make, opts, before, after, steps", [
    ("dam", dict(), 0, (8,), LANES * STEPS),
    ("dam", dict(), 3, (3,), LANES * STEPS),
    ("dam", dict(precision=1), 0, (8,), LANES * STEPS),
    ("batch", dict(precision=1), 2, (2,), LANES * STEPS),
    ("batch", dict(), 0, (1, 2, 4, 8), (GRIDS + LANES) * STEPS),
], ids=str)
def test_autotune(make, opts, before, after, steps):
    cfg, case, scenes = MAKE[make](**opts)
    s = vm.Solver(cfg, case)
    if scenes is not None:
        s.set_scenes(*scenes)
    assert s.init() == 0
    s.set_tuning(4, before)
    t = s.autotune(STEPS)
    assert t["cg_blocks_per_sm"] in after and s.get_tuning() == t
    assert s.scalar("steps") == steps
    s.close()
