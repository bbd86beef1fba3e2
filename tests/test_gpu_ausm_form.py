"""Orders 1 and 2 (AUSM+-up) at the states where the face pass's branches turn:
rest, low Mach numbers, transonic and supersonic faces of both signs, equal
neighbours (zero slopes), slopes of opposite signs and of very different size,
magnitudes whose reciprocals leave the fixed-point range, cut and solid cells,
odd box extents.  Against the oracle; per component 1e-12 of its domain
maximum, the tolerance of the other right-hand-side tests."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level, geometry
from helpers import rel_err
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# (at 1e-297 order 1 only: the reference's limiter has a guard of 1e-20 beside the slopes)
# order 2 reconstructs each component by itself: moderate jumps keep the face pressures positive
@pytest.mark.parametrize("n", [(1, 1, 1), (3, 2, 1), (33, 7, 10), (17, 40, 21)])
@pytest.mark.parametrize("kind,order,mach,scale", [
    (k, o, m, 1.0) for k, o in (("porous", 2), ("porous", 1), ("catalyst", 2), ("tg", 2)) for m in (0.0, 1e-3, 0.6, 1.0, 2.5)
] + [("sod", 1, 0.0, 1e-297), ("sod", 1, 0.0, 1e297), ("sod", 2, 0.0, 1e297)])
def test_rhs_and_fluxes(n, kind, order, mach, scale):
    P = {"tg": lambda: cases.taylor_green_mix(n=8), "catalyst": lambda: cases.catalyst(n=8),
         "porous": lambda: cases.porous_ib(n=8), "sod": lambda: cases.sod(n_cell=(8, 4, 4))}[kind]().params
    P.order_hyp = order
    rng = np.random.default_rng(sum(n) + int(10 * mach))
    g = abi.NGROW
    shape = tuple(q + 2 * g for q in n[::-1])
    vf = np.ones(shape)
    if kind in ("catalyst", "porous"):
        vf = rng.choice([0.0, 0.3, 0.8, 1.0], p=[0.05, 0.05, 0.05, 0.85], size=shape)

    def levels(spread):  # piecewise values with equal neighbours, plus slopes of 1e-12 to 1e-2
        return rng.choice(1.0 + spread * np.linspace(-1, 1, 5), size=shape) * (1.0 + 10.0 ** rng.uniform(-12, -2, shape))

    unit = 1.0 if kind == "sod" else 5.0
    spec = [levels(0.05) * unit for _ in range(P.nspec)]
    rho = spec[0] * P.molwt[0] if P.nspec == 1 else sum(spec[s] * P.molwt[s] for s in range(P.nspec))
    p = levels(0.05) * (1.0 if kind == "sod" else 1e5)
    c = np.sqrt(1.4 * p.mean() / rho.mean())
    signs = [-1.0, 0.0, 0.7, 1.0] if mach < 0.1 else [rng.choice([-1.0, 1.0])]
    vel = [mach * c * rng.choice(signs, size=shape) * levels(0.02) for _ in range(3)]
    S = cases.state_from_prim(P, rho, *vel, p, spec, vf)
    if scale != 1.0:  # density, momenta, energy, pressure and species scale together; speeds stay
        keep = [abi.VELX, abi.VELY, abi.VELZ, abi.TEMP, abi.VFRAC]
        S[[q for q in range(S.shape[0]) if q not in keep]] *= scale
    geom = geometry((0, 0, 0), [q - 1 for q in n], (0, 0, 0), [0.01 * q for q in n], (0, 0, 0))
    out = []
    for backend in ("numpy", "torch"):
        lev = Level([((0, 0, 0), tuple(q - 1 for q in n))], S.shape[0], backend=backend, device="cuda", with_flux=True)
        lev.set_sborder(0, S)
        if backend == "numpy":
            lib = oracle_lib.load("strict")
            assert lib.oracle_compute_dsdt(C.byref(P), C.byref(geom), lev.descriptors(), 1) == 0
        else:
            lib = abi.load()
            abi.check("mfg_init", lib.mfg_init(C.byref(P)))
            abi.check("dsdt", lib.mfg_compute_dsdt_flow(lev.descriptors(), 1, C.byref(geom), 0.0, 1e-6, None))
            torch.cuda.synchronize()
        out.append([lev.dsdt[0]] + lev.flux[0])
    for o, d in zip(*out):
        e, comp = rel_err(d.cpu().numpy(), o)
        assert e < 1e-12, (comp, e)
