"""Order 4 (central with dissipation) in its own kernel: regular faces, faces on
the solid side and first-order faces beside cut and solid cells, species that
are and are not advected, odd and smallest box extents, and the caller's flux
arrays.  Against the oracle; per component 1e-12 of its maximum, the tolerance
of the other right-hand-side tests."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level, geometry
from helpers import rel_err
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1, 1), (3, 2, 1), (33, 7, 10), (17, 40, 21)])
@pytest.mark.parametrize("kind", ["tg", "catalyst", "porous"])
def test_rhs_and_fluxes(n, kind):
    P = {"tg": lambda: cases.taylor_green_mix(n=8), "catalyst": lambda: cases.catalyst(n=8),
         "porous": lambda: cases.porous_ib(n=8)}[kind]().params
    P.order_hyp = 4
    rng = np.random.default_rng(sum(n))
    g = abi.NGROW
    shape = tuple(q + 2 * g for q in n[::-1])
    vf = np.ones(shape)
    if kind != "tg":
        vf = rng.choice([0.0, 0.3, 0.8, 1.0], p=[0.03, 0.03, 0.03, 0.91], size=shape)
    spec = [5.0 * (1.0 + 0.05 * rng.uniform(-1, 1, shape)) for _ in range(P.nspec)]
    rho = spec[0] * P.molwt[0] if P.nspec == 1 else sum(spec[s] * P.molwt[s] for s in range(P.nspec))
    p = 1e5 * (1.0 + 0.05 * rng.uniform(-1, 1, shape))
    c = np.sqrt(1.4 * p.mean() / rho.mean())
    vel = [0.3 * c * rng.uniform(-1, 1, shape) for _ in range(3)]
    S = cases.state_from_prim(P, rho, *vel, p, spec, vf)
    geom = geometry((0, 0, 0), [q - 1 for q in n], (0, 0, 0), [0.01 * q for q in n], (0, 0, 0))
    out = []
    for backend in ("numpy", "torch"):
        lev = Level([((0, 0, 0), tuple(q - 1 for q in n))], S.shape[0], backend=backend, device="cuda", with_flux=True)
        lev.set_sborder(0, S)
        if backend == "numpy":
            assert oracle_lib.load("strict").oracle_compute_dsdt(C.byref(P), C.byref(geom), lev.descriptors(), 1) == 0
            out.append((lev.dsdt[0], lev.flux[0]))
        else:
            gpu = abi.load()
            abi.check("init", gpu.mfg_init(C.byref(P)))
            st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
            abi.check("rhs", gpu.mfg_compute_dsdt_flow(lev.descriptors(), 1, C.byref(geom), 0.0, 1e-9, st))
            torch.cuda.synchronize()
            out.append((lev.dsdt[0].cpu().numpy(), [f.cpu().numpy() for f in lev.flux[0]]))
    (do, fo), (dg, fg) = out
    e, comp = rel_err(dg, do)
    assert e < 1e-12, (comp, e)
    for d in range(3):
        e, comp = rel_err(fg[d], fo[d])
        assert e < 1e-12, (d, comp, e)
