"""Order-5 right-hand side and face fluxes at the sizes where the column sweep
and the per-face form can go wrong: single cells, boxes shorter than the
stencil, extents around the sweep's segment length, many short columns, faces
on the solid side and first-order fallback faces in every position, and jumps
beyond 1e17 (where the two edge corrections are divided apart).  Against the
oracle; per component 1e-12 of its domain maximum, the tolerance of the other
right-hand-side tests."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level, geometry
from helpers import rel_err
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (2, 1, 5), (31, 3, 2), (32, 33, 4), (5, 34, 65), (64, 48, 33), (70, 9, 66)]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind,scale", [("tg", 1.0), ("catalyst", 1.0), ("sod", 1e18)])
def test_rhs_and_fluxes(n, kind, scale):
    P = {"tg": lambda: cases.taylor_green_mix(n=8), "catalyst": lambda: cases.catalyst(n=8),
         "sod": lambda: cases.sod(n_cell=(8, 4, 4))}[kind]().params
    rng = np.random.default_rng(sum(n))
    g = abi.NGROW
    shape = tuple(q + 2 * g for q in n[::-1])
    vf = np.ones(shape)
    if kind == "catalyst":  # cut, solid and gas cells in runs of a few cells
        vf = rng.choice([0.0, 0.3, 0.8, 1.0], p=[0.05, 0.03, 0.02, 0.9], size=shape)
    spec = [(1.0 + 0.2 * rng.random(shape)) * (scale if kind == "sod" else 5.0) for _ in range(P.nspec)]
    rho = sum(spec[s] * P.molwt[s] for s in range(P.nspec)) if kind != "sod" else spec[0] * P.molwt[0]
    p = (scale if kind == "sod" else 1e5) * (1.0 + 0.1 * rng.random(shape))
    c = np.sqrt(1.4 * p.mean() / rho.mean())
    vel = [0.3 * c * rng.standard_normal(shape) for _ in range(3)]
    S = cases.state_from_prim(P, rho, *vel, p, spec, vf)
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
