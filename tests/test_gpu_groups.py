"""The launches that serve several boxes at once: right-hand sides, stage
updates, bookends, norms and time-step estimates of lists of uneven boxes are
bitwise what the same boxes give one by one (every box keeps its own
arithmetic, scratch and partial sums), whatever the groups: single cells, thin
boxes, more boxes than a group holds, lists that end inside a group."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level
from helpers import perturb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# uneven boxes tiling 40 x 12 x 10 (x cuts, y cuts)
XCUT = [0, 1, 4, 5, 21, 33, 40]
YCUT = [0, 7, 12]


def uneven(nboxes):
    b = [((x0, y0, 0), (x1 - 1, y1 - 1, 9)) for y0, y1 in zip(YCUT, YCUT[1:]) for x0, x1 in zip(XCUT, XCUT[1:])]
    return b[:nboxes]


@pytest.mark.parametrize("nboxes", [1, 2, 7, 8, 9, 12])
@pytest.mark.parametrize("name,order", [("porous", 2), ("catalyst", 5), ("catalyst", 2), ("tg", 4)])
def test_group_equals_single_boxes(name, order, nboxes):
    c = {"porous": lambda: cases.porous_ib(n=40, order=order), "tg": lambda: cases.taylor_green_mix(n=40, order=order),
         "catalyst": lambda: cases.catalyst(n=40, order=order)}[name]()
    c = perturb(c, 3, vel_amp=1e-2)
    boxes = uneven(nboxes)
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
    rng = np.random.default_rng(nboxes)
    res = []
    for single in (False, True):
        lev = Level(boxes, c.ncomp, backend="torch", device="cuda", with_flux=True)
        for b, (lo, hi) in enumerate(boxes):
            pad = np.pad(c.state, [(0, 0)] + [(3, 3)] * 3, mode="edge")
            sl = (slice(None),) + tuple(slice(lo[q], hi[q] + 7) for q in (2, 1, 0))
            lev.set_sborder(b, pad[sl])
        lev.set_state(c.state)
        lev.set_state(c.state * (1.0 + 1e-6 * np.random.default_rng(5).standard_normal(c.state.shape)), which="old")
        d, g, st = lev.descriptors(), C.byref(c.geom), None
        calls = [(d, nboxes)] if not single else [(C.byref(d[b]), 1) for b in range(nboxes)]
        out = []
        for p, n in calls:
            abi.check("dsdt", lib.mfg_compute_dsdt_flow(p, n, g, 0.0, 1e-9, st))
        torch.cuda.synchronize()
        out += [x.cpu().numpy() for x in lev.dsdt] + [x.cpu().numpy() for f in lev.flux for x in f]
        for stage in (1, 2, 3):
            for p, n in calls:
                abi.check("stage", lib.mfg_rk3_stage(p, n, g, stage, 0.0, 1e-9, st))
            torch.cuda.synchronize()
            out += [x.cpu().numpy() for x in lev.s_new]
        est = []
        for p, n in calls:
            v = C.c_double()
            abi.check("est", lib.mfg_est_timestep(p, n, g, 0.0, C.byref(v), st))
            est.append(v.value)
        out.append(np.array(min(est)))
        res.append(out)
    for a, b in zip(*res):
        assert np.array_equal(a, b)


def test_level_step_does_not_depend_on_the_grouping():
    """mfg_advance_level over many small boxes, against mfg_boxlist_step's plain
    per-box launches of the same kernels; residual norms against the sums of
    the boxes' own."""
    c = perturb(cases.catalyst(n=20, order=5, max_grid=[7, 6, 20]), 9, vel_amp=1e-2)
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
    n = len(c.boxes)
    assert n > 8
    a = Level(c.boxes, c.ncomp, backend="torch", device="cuda")
    b = Level(c.boxes, c.ncomp, backend="torch", device="cuda")
    a.set_state(c.state)
    b.set_state(c.state)
    s = torch.cuda.Stream()
    st = C.c_void_p(s.cuda_stream)
    s.wait_stream(torch.cuda.current_stream())
    h = C.c_void_p()
    abi.check("create", lib.mfg_boxlist_create(b.descriptors(), n, (abi.Geom * 1)(c.geom), 1, C.byref(h)))
    rn = (C.c_double * c.ncomp)()
    dt = 2e-9
    for _ in range(2):
        abi.check("advance", lib.mfg_advance_level(a.descriptors(), n, C.byref(c.geom), 0.0, dt, 0, 1, rn, st))
        abi.check("plain", lib.mfg_boxlist_step(h, 0.0, dt, 0, st))
    s.synchronize()
    lib.mfg_boxlist_destroy(h)
    assert np.array_equal(a.get_state(c.shape_zyx), b.get_state(c.shape_zyx))
    one = (C.c_double * c.ncomp)()
    tot = np.zeros(c.ncomp)
    for q in range(n):
        abi.check("norms", lib.mfg_residual_norms(C.byref(a.descriptors()[q]), 1, dt, one, st))
        tot += np.array(one[:]) ** 2
    # the same squares, summed in another order: n boxes of up to 840 cells
    assert np.all(np.abs(np.array(rn[:]) - np.sqrt(tot)) <= 1e-13 * np.sqrt(tot))
