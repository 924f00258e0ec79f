"""mps_step_io above 65,536 particles, where u, v, w and p travel on a second stream beside
the neighbour search: the bits of mps_set_state + mps_step + mps_get_state with the host
state changed between the steps (so that the copied values, not the device's own, are
the ones used), and with fields left out of some steps' input (another set of fields
to apply, which a captured step has to follow)."""
import numpy as np
import pytest

import voxarmps_b200 as vm
from voxarmps_b200 import cases, config
from gpu_util import gpu_cfg

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "u", "v", "w", "p")


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("dim, fluid, tank", [
    (2, (253, 250), (300, 262)),     # 65,740
    (3, (31, 40, 27), (82, 61, 27)),  # 84,282
])
def test_equals_three_calls(dim, fluid, tank, graph):
    l0 = 0.01 if dim == 2 else 0.005
    case = cases.dam_break(dim, l0, fluid, tank)
    n = len(case["x"])
    assert n > 65_536
    cfg = config.reference_defaults(l0, dim)
    cfg.update(re_s=2.1 * l0, re_l=4.0 * l0, dt=1e-4 if dim == 2 else 5e-5, gy=-9.81)
    cfg = gpu_cfg(config.with_box(cfg, case))
    rng = np.random.default_rng(n)
    a, b = vm.Solver(cfg, case), vm.Solver(cfg, case)
    for s in (a, b):
        assert s.init() == 0
        s.set_graph(graph)
    ha = {k: np.zeros(n) for k in FIELDS}
    hb = {k: np.zeros(n) for k in FIELDS}
    for s, h in ((a, ha), (b, hb)):
        assert s.get_state(*[h[k].ctypes.data for k in FIELDS]) == 0
    fl = np.asarray(case["ptype"]) > 0
    left_out = {3: "p", 4: "uvw", 5: "uvwp"}
    for step in range(8):
        du = {k: rng.normal(0, 0.02, fl.sum()) for k in "uvw"[:dim]}
        for h in (ha, hb):
            for k in du:
                h[k][fl] += du[k]
            h["p"][fl] = h["p"][fl] * 0.9 + 50.0
        out = left_out.get(step, "")
        ins = [[0 if k in out else h[k].ctypes.data for k in FIELDS] for h in (ha, hb)]
        assert a.set_state(*ins[0]) == 0
        ra = a.step()
        assert a.get_state(*[ha[k].ctypes.data for k in FIELDS]) == 0
        rb = b.step_io(ins[1], [hb[k].ctypes.data for k in FIELDS])
        assert ra == rb == 0
        for k in FIELDS:
            assert np.array_equal(ha[k].view(np.uint64), hb[k].view(np.uint64)), (step, k)
    assert np.array_equal(a.get("pnew"), b.get("pnew"))
    a.close()
    b.close()
