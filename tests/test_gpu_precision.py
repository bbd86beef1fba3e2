"""Rounding errors against extended precision: the pressure of a mixture, and
fluxes whose exact value is plain (order 4 of a gas at rest, order 1 along lines of
constant state), have an rms error no larger than the reference's own order of
operations in double precision (the oracle's)."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level, geometry
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = abi.NGROW
L = np.longdouble
N = (40, 36, 30)


def params(name, order=5):
    P = {"five": lambda: cases.taylor_green_mix(n=8, order=order), "ten": lambda: cases.catalyst(n=8, order=order),
         "background": lambda: cases.catalyst(n=8, order=order, bg_gas=True),
         "one": lambda: cases.porous_ib(n=8, order=order)}[name]().params
    P.visc_gas = P.cond_gas = P.visc_solid = P.cond_solid = 0.0
    return P


def state(P, shape, rng, vel):
    spec = [5.0 * rng.gamma(4.0, 0.25, shape) for _ in range(P.nspec)]
    rho = sum(spec[s] * (P.molwt[s] or 1.0) for s in range(P.nspec))
    if P.thermo_kind == abi.THERMO_BG_GAS:
        rho = rho + 20.0 * P.bg_molwt
    return cases.state_from_prim(P, rho, *vel, 1e5 * rng.uniform(0.9, 1.1, shape), spec, np.ones(shape))


def pressure(P, S):
    S = L(S)
    rhoe = S[abi.RHOE] - (S[abi.RHOU] ** 2 + S[abi.RHOV] ** 2 + S[abi.RHOW] ** 2) / (2 * S[abi.RHO])
    if P.thermo_kind == abi.THERMO_MASS_SINGLE:
        return rhoe * (L(P.gamma_single) - 1)
    c = [S[abi.FLO_NVARS + s] for s in range(P.ngas)]
    if P.thermo_kind == abi.THERMO_BG_GAS:
        c.append((S[abi.RHO] - sum(x * L(P.molwt[s]) for s, x in enumerate(c))) / L(P.bg_molwt))
    return rhoe * sum(c) / sum(x / (L(P.gamma[s]) - 1) for s, x in enumerate(c))


def rms(x, ref):
    return float(np.sqrt(np.mean((((L(x) - ref) / ref)) ** 2)))


def run(P, S, n, call):
    """Level of both backends with S (grown) in sborder and s_new."""
    geom = geometry((0, 0, 0), [q - 1 for q in n], (0, 0, 0), [0.01 * q for q in n], (0, 0, 0))
    out = []
    for backend in ("numpy", "torch"):
        lev = Level([((0, 0, 0), tuple(q - 1 for q in n))], S.shape[0], backend=backend, device="cuda", with_flux=True)
        lev.set_sborder(0, S)
        lev.set_state(S[:, G:-G, G:-G, G:-G])
        lib = oracle_lib.load("strict") if backend == "numpy" else abi.load()
        if backend == "torch":
            abi.check("mfg_init", lib.mfg_init(C.byref(P)))
        assert call(lib, backend == "numpy", lev.descriptors(), geom) == 0
        torch.cuda.synchronize()
        out.append(lev)
    return out


@pytest.mark.parametrize("name", ["five", "ten", "background"])
def test_pressure(name):
    P, rng = params(name), np.random.default_rng(1)
    shape = tuple(q + 2 * G for q in N[::-1])
    S = state(P, shape, rng, [40.0 * rng.standard_normal(shape) for _ in range(3)])

    def call(lib, oracle, d, g):
        return lib.oracle_update_primitive_vars(C.byref(P), d, 1) if oracle else \
            lib.mfg_update_primitive_vars(d, 1, C.byref(g), None)

    o, k = (x.get_state(N[::-1])[abi.PRES] for x in run(P, S, N, call))
    ref = pressure(P, S[:, G:-G, G:-G, G:-G])
    print(name, rms(o, ref) / 2.0 ** -53, rms(k, ref) / 2.0 ** -53)
    assert rms(k, ref) <= rms(o, ref)


def rhs(P):
    return lambda lib, oracle, d, g: lib.oracle_compute_dsdt(C.byref(P), C.byref(g), d, 1) if oracle else \
        lib.mfg_compute_dsdt_flow(d, 1, C.byref(g), 0.0, 1e-6, None)


@pytest.mark.parametrize("name", ["five", "one"])
def test_order4_momentum_at_rest(name):
    P, rng = params(name, 4), np.random.default_rng(2)
    shape = tuple(q + 2 * G for q in N[::-1])
    S = state(P, shape, rng, [np.zeros(shape)] * 3)
    o, k = run(P, S, N, rhs(P))
    p = pressure(P, S)
    for d in range(3):
        ax = 2 - d
        f = [np.moveaxis(p[tuple(slice(None) if a == ax else slice(G, -G) for a in range(3))], ax, -1)[..., G - 2 + q:]
             for q in range(4)]
        m = N[d] + 1
        ref = L(0.08333333333) * (7 * (f[1][..., :m] + f[2][..., :m]) - f[0][..., :m] - f[3][..., :m])
        x, y = (np.moveaxis(np.asarray(v.flux[0][d][abi.RHOU + d].cpu() if v is k else v.flux[0][d][abi.RHOU + d]), ax, -1)
                for v in (o, k))
        print(name, d, rms(x, ref) / 2.0 ** -53, rms(y, ref) / 2.0 ** -53)
        assert rms(y, ref) <= rms(x, ref)


@pytest.mark.parametrize("name", ["five", "one"])
@pytest.mark.parametrize("d", [0, 1, 2])
def test_order1_momentum_of_constant_lines(name, d):
    """Both sides of a face alike: the flux of the normal momentum is rho v^2 + p."""
    P, rng = params(name, 1), np.random.default_rng(3)
    shape = tuple(q + 2 * G for q in N[::-1])
    S = state(P, shape, rng, [100.0 * rng.standard_normal(shape) for _ in range(3)])
    ax = 3 - d
    S = np.repeat(np.take(S, [0], axis=ax), S.shape[ax], axis=ax)
    S[abi.VELX:abi.VELZ + 1] = 0.0  # no viscous terms
    o, k = run(P, S, N, rhs(P))
    one = tuple(slice(0, 1) if a == ax - 1 else slice(G, -G) for a in range(3))
    ref = pressure(P, S)[one] + L(S[abi.RHOU + d][one]) ** 2 / S[abi.RHO][one]
    x, y = (np.take(np.asarray(v.flux[0][d][abi.RHOU + d].cpu() if v is k else v.flux[0][d][abi.RHOU + d]), [1], axis=ax - 1)
            for v in (o, k))
    print(name, d, rms(x, ref) / 2.0 ** -53, rms(y, ref) / 2.0 ** -53)
    assert rms(y, ref) <= rms(x, ref)
