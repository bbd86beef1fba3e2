"""The search over tiles of a box list runs the step's own kernels, each phase on
what the one before wrote: on a list that has run no step it leaves the fluxes
and rates of its state, bitwise those of the per-box calls, and no status."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level
from helpers import perturb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [5, 4, 2])
def test_autotune_leaves_the_rates_of_its_state(order):
    c = perturb(cases.catalyst(n=24, order=order, max_grid=12), 21, vel_amp=1e-2)
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
    s = torch.cuda.Stream()
    st = C.c_void_p(s.cuda_stream)
    n = len(c.boxes)
    lev = [Level(c.boxes, c.ncomp, backend="torch", device="cuda", with_flux=True) for _ in range(2)]
    for x in lev:
        x.set_state(c.state)
        for q in x.dsdt + [f for b in x.flux for f in b]:
            q.fill_(-1.0)
    torch.cuda.synchronize()
    h = C.c_void_p()
    abi.check("create", lib.mfg_boxlist_create(lev[0].descriptors(), n, (abi.Geom * 1)(c.geom), 1, C.byref(h)))
    with torch.cuda.stream(s):
        abi.check("autotune", lib.mfg_boxlist_autotune(h, 2e-9, (C.c_double * 16)(), st))
        d, g = lev[1].descriptors(), C.byref(c.geom)
        abi.check("fill", lib.mfg_fill_patch(d, n, g, 1, 0.0, st))
        abi.check("cut", lib.mfg_cutcells(d, n, g, 0.0, st))
        abi.check("dsdt", lib.mfg_compute_dsdt_flow(d, n, g, 0.0, 2e-9, st))
    s.synchronize()
    lib.mfg_boxlist_destroy(h)
    status = C.c_uint()
    abi.check("status", lib.mfg_status(C.byref(status), 1))
    assert status.value == 0
    for b in range(n):
        for x, y in zip([lev[0].dsdt[b]] + lev[0].flux[b], [lev[1].dsdt[b]] + lev[1].flux[b]):
            assert np.array_equal(x.cpu().numpy(), y.cpu().numpy()), b
