"""Values at the ends of the range where the kernels refine a hardware
approximation in place of a division or a square root: an infinite energy gives
an infinite temperature and pressure, and a pressure of subnormal size a finite
right-hand side, as the oracle's."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level, geometry
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = abi.NGROW


def case(name):
    return {"molar": lambda: cases.taylor_green_mix(n=8), "bg": lambda: cases.catalyst(n=8, bg_gas=True),
            "mass": lambda: cases.sod(n_cell=(8, 4, 4))}[name]()


@pytest.mark.parametrize("name", ["molar", "bg", "mass"])
def test_infinite_energy(name):
    c = case(name)
    S = c.state.copy()
    S[abi.VFRAC] = 1.0
    S[abi.RHOE].flat[::3] = np.inf
    S[abi.RHOE].flat[1::3] *= 1e160 / np.abs(S[abi.RHOE]).flat[1]
    shape = S.shape[1:]
    box = [((0, 0, 0), tuple(q - 1 for q in shape[::-1]))]
    out = []
    for backend in ("numpy", "torch"):
        lev = Level(box, S.shape[0], backend=backend, device="cuda")
        lev.set_state(S)
        if backend == "numpy":
            lib = oracle_lib.load("strict")
            assert lib.oracle_update_primitive_vars(C.byref(c.params), lev.descriptors(), 1) == 0
        else:
            lib = abi.load()
            abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
            abi.check("prims", lib.mfg_update_primitive_vars(lev.descriptors(), 1, C.byref(c.geom), None))
        out.append(lev.get_state(shape))
    o, d = out
    for q in (abi.PRES, abi.TEMP):
        assert np.all(np.isposinf(o[q].flat[::3])) and np.all(np.isposinf(d[q].flat[::3])), q
        assert np.all(np.abs(d[q].flat[1::3] / o[q].flat[1::3] - 1.0) < 1e-14), q


@pytest.mark.parametrize("order", [4, 5])
def test_subnormal_pressure(order):
    P = cases.taylor_green_mix(n=8, order=order).params
    n = (6, 5, 4)
    shape = tuple(q + 2 * G for q in n[::-1])
    rng = np.random.default_rng(order)
    spec = [1.0 + 0.1 * rng.random(shape) for _ in range(P.nspec)]
    rho = sum(spec[s] * P.molwt[s] for s in range(P.nspec))
    zero = np.zeros(shape)
    S = cases.state_from_prim(P, rho, zero, zero, zero, 1e-311 * (1.0 + rng.random(shape)), spec, np.ones(shape))
    geom = geometry((0, 0, 0), [q - 1 for q in n], (0, 0, 0), [0.01 * q for q in n], (0, 0, 0))
    out = []
    for backend in ("numpy", "torch"):
        lev = Level([((0, 0, 0), tuple(q - 1 for q in n))], S.shape[0], backend=backend, device="cuda")
        lev.set_sborder(0, S)
        if backend == "numpy":
            assert oracle_lib.load("strict").oracle_compute_dsdt(C.byref(P), C.byref(geom), lev.descriptors(), 1) == 0
        else:
            lib = abi.load()
            abi.check("mfg_init", lib.mfg_init(C.byref(P)))
            abi.check("dsdt", lib.mfg_compute_dsdt_flow(lev.descriptors(), 1, C.byref(geom), 0.0, 1e-6, None))
            torch.cuda.synchronize()
        out.append(np.asarray(lev.dsdt[0].cpu() if backend == "torch" else lev.dsdt[0]))
    assert np.all(np.isfinite(out[0])) and np.all(np.isfinite(out[1]))
    for s in range(P.nspec):  # diffusion: the only flux of ordinary size
        a, b = (x[abi.FLO_NVARS + s] for x in out)
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
