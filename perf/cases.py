"""What a user of this framework has it do, as cases that can be timed and compared.

The work is the explicit right-hand side and SSP-RK3 step of a box list and
what is built on it: whole coarse steps of one level (time-step estimate,
step, residual norms) on the four flow families of mesoflow_gb300.cases, the
same step on a state kept in host memory, the right-hand side alone on one box
with its face fluxes (what an AMReX driver calls per box), the subcycled
multi-level step, the implicit chemistry sub-step and the adjoint gradient.

  kind "step"     mfg_est_timestep + mfg_advance_level (norms on): one pass of
                  mflo::EvolveAMR's loop on one level
  kind "host"     mfg_advance_level_host on pinned host buffers
  kind "rhs"      mfg_compute_dsdt_flow on one grown box, with face fluxes
  kind "amr"      mfg_boxlist_step_amr, replayed from its CUDA graph
  kind "chem"     mfg_chem_substep with the implicit integrator
  kind "adjoint"  ReactionProblem.gradient

Flow families: "sod" (single gas, shock tube), "tg" (five-species
Taylor-Green), "porous" (air through a sphere pack, immersed boundary),
"catalyst" (8 gas + 2 site species, immersed catalyst, surface chemistry).
Steps advance the state they are given, as a simulation does.
"""
import ctypes as C
import math

import numpy as np
import torch

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.adjoint import ReactionProblem
from mesoflow_gb300.level import Level, MultiLevel, chop, geometry

G = abi.NGROW
NF = abi.FLO_NVARS
RHO, RHOU, RHOE, DENS, VELX, PRES, TEMP, VFRAC = (abi.RHO, abi.RHOU, abi.RHOE, abi.DENS, abi.VELX, abi.PRES,
                                                  abi.TEMP, abi.VFRAC)
NSPEC = {"sod": 1, "tg": 5, "porous": 1, "catalyst": 10}
DX = {"porous": 2e-6, "catalyst": 1e-5}


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one finely refined box of an AMR hierarchy, right-hand side and fluxes for the
        # flux registers: the smallest call a driver makes, latency and launches count
        {"name": "rhs_box16_weno", "kind": "rhs", "flow": "catalyst", "nx": 16, "ny": 16, "nz": 16, "order": 5},
        # shock-tube verification run, 4096 cells: the smallest whole step
        {"name": "step_sod_256x4x4", "kind": "step", "flow": "sod", "nx": 256, "ny": 4, "nz": 4, "order": 5,
         "max_grid": 64},
        # one large multi-species box, the default scheme (AUSM+-up with MUSCL), ragged extents
        {"name": "rhs_ausm_61x47x38", "kind": "rhs", "flow": "catalyst", "nx": 61, "ny": 47, "nz": 38, "order": 2},
        # central scheme with dissipation (smooth turbulence runs), ragged extents
        {"name": "rhs_central_57x64x33", "kind": "rhs", "flow": "tg", "nx": 57, "ny": 64, "nz": 33, "order": 4},
        # the box of the turbulence configuration
        {"name": "rhs_weno_64", "kind": "rhs", "flow": "tg", "nx": 64, "ny": 64, "nz": 64, "order": 5},
        # pore-scale flow on a domain whose extents do not divide by the box size
        {"name": "step_porous_100x76x52", "kind": "step", "flow": "porous", "nx": 100, "ny": 76, "nz": 52, "order": 2,
         "max_grid": 32},
        # reacting catalyst block: immersed boundary, ten species, surface chemistry
        {"name": "step_catalyst_64", "kind": "step", "flow": "catalyst", "nx": 64, "ny": 64, "nz": 64, "order": 5,
         "max_grid": 32},
        # turbulent mixing, five species
        {"name": "step_tg_128", "kind": "step", "flow": "tg", "nx": 128, "ny": 128, "nz": 128, "order": 5,
         "max_grid": 64},
        # pore-scale flow for a driver that keeps its state in host memory
        {"name": "host_porous_128", "kind": "host", "flow": "porous", "nx": 128, "ny": 128, "nz": 128, "order": 2,
         "max_grid": 64},
        # the pore-scale production size (bench.py's workload)
        {"name": "step_porous_256", "kind": "step", "flow": "porous", "nx": 256, "ny": 256, "nz": 256, "order": 2,
         "max_grid": 64},
        # three refinement levels around a catalyst surface, subcycled coarse step
        {"name": "amr_catalyst_3lev", "kind": "amr", "flow": "catalyst", "n0": 32, "nlev": 3, "order": 5,
         "nspheres": 6, "shape": 4},
        # kinetics fit: gradient of the surface reaction rate through ten steps
        {"name": "adjoint_catalyst_32", "kind": "adjoint", "flow": "catalyst", "n": 32, "nsteps": 10, "every": 5},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "step", "step", "step", "host", "chem", "amr", "adjoint"])
    flow = rng.choice(["sod", "tg", "porous", "catalyst"])
    if kind == "rhs":
        return {"kind": kind, "flow": flow, "nx": _log(rng, 8, 80), "ny": _log(rng, 8, 80), "nz": _log(rng, 8, 80),
                "order": rng.choice([1, 2, 2, 4, 5, 5, 5])}
    if kind in ("step", "host"):
        order = {"sod": 5, "tg": 5, "porous": rng.choice([2, 2, 5]), "catalyst": rng.choice([2, 5, 5])}[flow]
        n = [_log(rng, 16, 160 if order == 2 else 96) for _ in range(3)]
        if flow == "sod":
            n = [_log(rng, 64, 512), rng.choice([4, 6, 8]), rng.choice([4, 6, 8])]
        return {"kind": kind, "flow": flow, "nx": n[0], "ny": n[1], "nz": n[2], "order": order,
                "max_grid": rng.choice([16, 32, 64])}
    if kind == "chem":
        return {"kind": kind, "flow": "catalyst", "nx": _log(rng, 8, 48), "ny": _log(rng, 8, 48),
                "nz": _log(rng, 8, 48), "order": 5}
    if kind == "amr":
        n0 = rng.choice([32, 48])
        return {"kind": kind, "flow": "catalyst", "n0": n0, "nlev": 2 if n0 > 32 else rng.choice([2, 3]),
                "order": rng.choice([2, 5]), "nspheres": rng.randint(3, 9), "shape": rng.randint(1, 99)}
    return {"kind": "adjoint", "flow": "catalyst", "n": rng.choice([16, 24, 32]), "nsteps": rng.randint(4, 10),
            "every": rng.choice([0, 4, 5])}


# ---------------------------------------------------------------------------
# set-up: parameter tables, geometry and seeded flow fields
# ---------------------------------------------------------------------------
def _params(case):
    base = {"sod": lambda: cases.sod(n_cell=(8, 4, 4)), "tg": lambda: cases.taylor_green_mix(n=8),
            "porous": lambda: cases.porous_ib(n=8), "catalyst": lambda: cases.catalyst(n=8)}[case["flow"]]()
    base.params.order_hyp = case["order"]
    # three-dimensional acoustic limit with a margin, as models/porousParticle/inputs has it
    base.params.cfl = 0.1 if case["flow"] in DX else 0.2
    return base.params


def _geom(flow, n):
    if flow == "sod":
        return geometry((0, 0, 0), [q - 1 for q in n], (0, 0, 0), (1.0, 0.125, 0.125), (0, 1, 1))
    if flow == "tg":
        return geometry((0, 0, 0), [q - 1 for q in n], (-1, -1, -1), (1, 1, 1), (1, 1, 1))
    d = DX[flow]
    return geometry((0, 0, 0), [q - 1 for q in n], (0, 0, 0), [q * d for q in n], (0, 0, 0))


_VF = {}


def _vfrac(flow, n):
    """Immersed solid of an n = (nx, ny, nz) region (the same one for every seed:
    a user's geometry file), kept because it is made on the host."""
    key = (flow, tuple(n))
    if key not in _VF:
        m = max(n)
        if flow == "porous":
            vf = cases.sphere_pack_vfrac(m, 3, 0.4)
        else:
            vf = cases.sphere_pack_vfrac(m, 5, 0.15, rmin=max(2.0, m / 64), rmax=max(4.0, m / 20))
            q = m // 3
            vf[q:2 * q, m // 4:3 * m // 4, m // 4:3 * m // 4] = 0.0
        if len(_VF) > 8:
            _VF.clear()
        _VF[key] = np.ascontiguousarray(vf[:n[2], :n[1], :n[0]])
    return torch.as_tensor(_VF[key], device="cuda")


def _thermo_p(P, rhoe, rho, spec):
    if P.thermo_kind == abi.THERMO_MASS_SINGLE:
        return rhoe * (P.gamma_single - 1.0)
    cvs = sum(P.R_univ / (P.gamma[s] - 1.0) * spec[s] for s in range(P.ngas))
    T = rhoe / cvs
    return sum(spec[s] * P.R_univ * T for s in range(P.ngas))


def _thermo_t(P, rho, p, spec):
    if P.thermo_kind == abi.THERMO_MASS_SINGLE:
        return p / P.gas_R / rho
    return p / (sum(spec[s] for s in range(P.ngas)) * P.R_univ)


def _thermo_gamma(P, rho, spec):
    if P.thermo_kind == abi.THERMO_MASS_SINGLE:
        return torch.full_like(rho, P.gamma_single)
    tot = sum(spec[s] for s in range(P.ngas))
    return 1.0 + 1.0 / sum(spec[s] / tot / (P.gamma[s] - 1.0) for s in range(P.ngas))


def _thermo_e(P, rho, p, spec):
    if P.thermo_kind == abi.THERMO_MASS_SINGLE:
        return p / (P.gamma_single - 1.0) / rho
    T = _thermo_t(P, rho, p, spec)
    if P.energy_form == abi.EFORM_MASS_CV:
        tot = sum(spec[s] for s in range(P.ngas))
        return T * sum(P.R_univ / (P.gamma[s] - 1.0) / P.molwt[s] * (spec[s] / tot) for s in range(P.ngas))
    return T * sum(P.R_univ / (P.gamma[s] - 1.0) * spec[s] for s in range(P.ngas)) / rho


def _from_prim(P, rho, vel, p, spec, vf):
    S = torch.empty((NF + P.nspec,) + tuple(rho.shape), dtype=torch.float64, device="cuda")
    S[RHO], S[DENS], S[PRES], S[VFRAC] = rho, rho, p, vf
    for a in range(3):
        S[RHOU + a], S[VELX + a] = rho * vel[a], vel[a]
    S[TEMP] = _thermo_t(P, rho, p, spec)
    S[RHOE] = rho * _thermo_e(P, rho, p, spec) + 0.5 * rho * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)
    for s in range(P.nspec):
        S[NF + s] = spec[s]
    return S


def _flow(case, P, n, seed):
    """Seeded flow field (ncomp, nz, ny, nx) of the case's family on n cells:
    the family's mean flow with fluctuations."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    shape = (n[2], n[1], n[0])
    noise = lambda: torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")  # noqa: E731
    ax = [(torch.arange(q, dtype=torch.float64, device="cuda") + 0.5) / q for q in n]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    one = torch.ones(shape, dtype=torch.float64, device="cuda")
    flow = case["flow"]
    if flow == "sod":
        left = (X < 0.5).expand(shape)
        rho = torch.where(left, one, 0.125 * one) * (1 + 1e-3 * noise())
        p = torch.where(left, one, 0.1 * one) * (1 + 1e-3 * noise())
        vel = [1e-2 * noise() for _ in range(3)]
        return _from_prim(P, rho, vel, p, [rho / P.molwt[0]], one)
    if flow == "tg":
        x, y, z = math.pi * (2 * X - 1), math.pi * (2 * Y - 1), math.pi * (2 * Z - 1)
        vel = [10 * torch.sin(x) * torch.cos(y) * torch.cos(z) + 0.1 * noise(),
               -10 * torch.cos(x) * torch.sin(y) * torch.cos(z) + 0.1 * noise(), 0.1 * noise()]
        u = torch.rand((P.nspec, 2) + shape, generator=gen, dtype=torch.float64, device="cuda")
        g = -torch.log(u[:, 0] * u[:, 1] + 1e-300)  # Gamma(2): mass fractions are Dirichlet(2)
        yk = g / g.sum(0)
        p = 1e5 * one
        rho = p / (P.R_univ * 300.0 * sum(yk[s] / P.molwt[s] for s in range(P.nspec)))
        return _from_prim(P, rho, vel, p, [rho * yk[s] / P.molwt[s] for s in range(P.nspec)], one)
    vf = _vfrac(flow, n)
    if flow == "porous":
        p = 1e5 * (1 + 1e-3 * (1 - X)) * (1 + 2e-4 * noise())
        rho = p / (P.gas_R * 300.0 * (1 + 1e-3 * noise()))
        vel = [vf * ((0.05 if a == 0 else 0.0) + 0.01 * noise()) for a in range(3)]
        return _from_prim(P, rho, vel, p, [rho / P.molwt[0]], vf)
    ctot = 1e5 / (P.R_univ * 500.0)
    frac = [0.7, 0.1, 0.05, 0.05, 0.04, 0.03, 0.02, 0.01]
    spec = [ctot * frac[s] * (1 + 1e-2 * noise()) for s in range(P.ngas)]
    p = P.R_univ * 500.0 * (1 + 1e-3 * noise()) * sum(spec)
    rho = sum(spec[s] * P.molwt[s] for s in range(P.ngas))
    site = torch.where(vf < 1.0, 50.0 * one, 0.0 * one)
    fluid = torch.where(vf == 1.0, one, 0.0 * one)
    vel = [fluid * ((1.0 if a == 0 else 0.0) + 0.01 * noise()) for a in range(3)]
    return _from_prim(P, rho, vel, p, spec + [0.6 * site, 0.4 * site], vf)


class _State:
    """What the user's program keeps: arrays, descriptors, handles."""

    def __init__(self):
        self.lib = abi.load()
        self.handle = None
        self.stream = torch.cuda.current_stream()
        abi.check("mfg_status", self.lib.mfg_status(C.byref(C.c_uint32()), 1))

    def st(self):
        return C.c_void_p(self.stream.cuda_stream)

    def __del__(self):
        if self.handle is not None:
            torch.cuda.synchronize()
            self.lib.mfg_boxlist_destroy(self.handle)
            self.handle = None


def _cells3(case):
    return [case["nx"], case["ny"], case["nz"]]


def _set_chem(lib, kind):
    abi.check("mfg_set_chem_integrator", lib.mfg_set_chem_integrator(kind, 1e-8, 1e-12, 1000))


def _level_state(case, seed):
    s = _State()
    P = _params(case)
    n = _cells3(case)
    _set_chem(s.lib, 0)
    abi.check("mfg_init", s.lib.mfg_init(C.byref(P)))
    s.geom = _geom(case["flow"], n)
    boxes = chop((0, 0, 0), [q - 1 for q in n], case["max_grid"])
    s.level = Level(boxes, NF + P.nspec, backend="torch", device="cuda", with_dsdt=False)
    S = _flow(case, P, n, seed)
    # phi_new of all boxes in one allocation (the boxes one after the other)
    s.flat = torch.empty(S.numel(), dtype=torch.float64, device="cuda")
    at = 0
    for b, (lo, hi) in enumerate(boxes):
        old = s.level.s_new[b]
        view = s.flat[at:at + old.numel()].view(old.shape)
        at += old.numel()
        view.copy_(S[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1])
        s.level.s_new[b] = view
    s.desc = s.level.descriptors()
    s.nbox = len(boxes)
    s.norms = (C.c_double * (NF + P.nspec))()
    s.time = 0.0
    return s


def _est(s):
    dt = C.c_double()
    abi.check("mfg_est_timestep", s.lib.mfg_est_timestep(s.desc, s.nbox, C.byref(s.geom), s.time, C.byref(dt), s.st()))
    return dt.value


def _amr_case(case):
    return cases.catalyst_amr(n0=case["n0"], nlev=case["nlev"], order=case["order"], seed=case["shape"], blocking=8,
                              max_grid=16, base_grid=16, nspheres=case["nspheres"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return ("step", _level_state(case, seed))
    if kind == "host":
        s = _level_state(case, seed)
        s.dt = _est(s)
        # the driver's own FABs: pinned host arrays, one after the other
        s.host = torch.empty(s.flat.numel(), dtype=torch.float64).pin_memory()
        s.host.copy_(s.flat)
        parts, at = [], 0
        for a in s.level.s_new:
            parts.append(s.host[at:at + a.numel()].view(a.shape))
            at += a.numel()
        s.views = s.level.host_views(parts)
        torch.cuda.synchronize()
        return ("host", s)
    if kind == "amr":
        s = _State()
        amr = _amr_case(case)
        rng = np.random.default_rng(seed)
        for a in amr.states:
            g = a[NF:NF + 8]
            g *= 1.0 + 1e-3 * rng.standard_normal(g.shape)
        _set_chem(s.lib, 0)
        abi.check("mfg_init", s.lib.mfg_init(C.byref(amr.params)))
        s.ml = MultiLevel(amr, backend="torch", device="cuda")
        # phi_new of every box of every level in one allocation
        s.flat = torch.empty(sum(a.size for a in amr.states), dtype=torch.float64, device="cuda")
        at = 0
        for lv, b in s.ml.index:
            old = s.ml.levels[lv].s_new[b]
            view = s.flat[at:at + old.numel()].view(old.shape)
            at += old.numel()
            view.copy_(old)
            s.ml.levels[lv].s_new[b] = view
        s.handle = C.c_void_p()
        s.desc, s.geoms = s.ml.descriptors(), s.ml.geoms()
        abi.check("mfg_boxlist_create", s.lib.mfg_boxlist_create(s.desc, len(amr.boxes), s.geoms, len(amr.geoms),
                                                                 C.byref(s.handle)))
        s.stream = torch.cuda.Stream()  # graphs are captured on a stream of their own
        s.stream.wait_stream(torch.cuda.current_stream())
        s.time = 0.0
        return ("amr", s)
    if kind == "adjoint":
        n = case["n"]
        c = cases.catalyst(n=n, order=5, max_grid=16 if n % 16 == 0 else 8, seed=5)
        rng = np.random.default_rng(seed)
        c.state[NF:NF + 8] *= 1.0 + 1e-3 * rng.standard_normal(c.state[NF:NF + 8].shape)
        for r in range(c.params.nreact):  # rate constants of 1e3 at 500 K: every reaction carries weight
            c.params.A[r] = 1e3 * math.exp(c.params.Ea[r] / (cases.RU * 500.0))
        s = _State()
        _set_chem(s.lib, 0)
        s.problem = ReactionProblem(c, case["nsteps"], 4e-9, checkpoint_every=case["every"])
        s.logA = np.array([math.log(c.params.A[r]) for r in range(c.params.nreact)])
        s.u_in = c.meta["u_in"]
        return ("adjoint", s)
    s = _State()
    P = _params(case)
    n = _cells3(case)
    _set_chem(s.lib, 1 if kind == "chem" else 0)
    if kind == "chem":
        for r in range(P.nreact):  # a stiff table: rate constants of 1e3 to 1e6 at 500 K
            P.A[r] = 10.0 ** (3 + 3 * (r % 4) / 3.0) * math.exp(P.Ea[r] / (cases.RU * 500.0))
    abi.check("mfg_init", s.lib.mfg_init(C.byref(P)))
    s.geom = _geom(case["flow"], n)
    box = [((0, 0, 0), tuple(q - 1 for q in n))]
    s.level = Level(box, NF + P.nspec, backend="torch", device="cuda", with_dsdt=kind == "rhs", with_flux=kind == "rhs",
                    with_sborder=kind == "rhs")
    if kind == "rhs":
        s.level.sborder[0].copy_(_flow(case, P, [q + 2 * G for q in n], seed))
    else:
        s.level.s_old[0].copy_(_flow(case, P, n, seed))
    s.desc = s.level.descriptors()
    return (kind, s)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind, s = state
    if kind == "step":
        dt = _est(s)
        abi.check("mfg_advance_level", s.lib.mfg_advance_level(s.desc, s.nbox, C.byref(s.geom), s.time, dt, 0, 1,
                                                               s.norms, s.st()))
        s.time += dt
        return {"state": s.flat, "norms": np.array(s.norms[:]), "dt": np.array([dt])}
    if kind == "host":
        abi.check("mfg_advance_level_host", s.lib.mfg_advance_level_host(
            s.desc, s.nbox, C.byref(s.geom), s.time, s.dt, 0, 1, s.views, s.norms, s.st()))
        s.time += s.dt
        return {"state": s.host, "norms": np.array(s.norms[:])}
    if kind == "rhs":
        abi.check("mfg_compute_dsdt_flow", s.lib.mfg_compute_dsdt_flow(s.desc, 1, C.byref(s.geom), 0.0, 1e-9, s.st()))
        return {"dsdt": list(s.level.dsdt[0].unbind(0)), "flux": s.level.flux[0]}
    if kind == "amr":
        abi.check("mfg_boxlist_step_amr", s.lib.mfg_boxlist_step_amr(s.handle, s.time, 4e-9, 2, s.st()))
        s.time += 4e-9
        return s.flat
    if kind == "chem":
        abi.check("mfg_chem_substep", s.lib.mfg_chem_substep(s.desc, 1, C.byref(s.geom), 0.0, 1e-6, s.st()))
        return s.level.s_new[0]
    J, gA, gu = s.problem.gradient(s.logA, s.u_in)
    return {"J": np.array([J]), "dlogA": gA, "du_in": np.array([gu])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _rhs_flops(flow, order):
    """FP64 operations per cell of one right-hand side: per face and component
    the reconstruction and flux, per face the scheme's scalars and the viscous
    terms, three faces per cell (a fused multiply-add counts two)."""
    c = 5 + NSPEC[flow]
    per_comp = {1: 6, 2: 16, 4: 20, 5: 150}[order]
    per_face = {1: 120, 2: 120, 4: 60, 5: 60}[order]
    return 3 * (c * per_comp + per_face) + 8 * c + 40


def work(case):
    kind = case["kind"]
    if kind in ("step", "host", "rhs", "chem"):
        N = NF + NSPEC[case["flow"]]
        n = _cells3(case)
        cells = n[0] * n[1] * n[2]
        f = _rhs_flops(case["flow"], case["order"])
        if kind == "rhs":
            grown = (n[0] + 6) * (n[1] + 6) * (n[2] + 6)
            faces = sum((n[0] + (d == 0)) * (n[1] + (d == 1)) * (n[2] + (d == 2)) for d in range(3))
            return {"bytes": 8 * N * (grown + cells + faces), "flops": f * cells}
        if kind == "chem":
            return {"bytes": 16 * N * cells, "flops": 2000 * cells}
        return {"bytes": 16 * N * cells, "flops": (3 * f + 10 * N) * cells}
    N = NF + NSPEC["catalyst"]
    f = 3 * _rhs_flops("catalyst", 5) + 10 * N
    if kind == "amr":
        if case["order"] == 2:
            f = 3 * _rhs_flops("catalyst", 2) + 10 * N
        cells, steps = 0, 0
        for lo, hi, lv in _amr_case(case).boxes:
            m = math.prod(hi[d] - lo[d] + 1 for d in range(3))
            cells += m
            steps += m * 2 ** lv
        return {"bytes": 16 * N * cells, "flops": f * steps}
    cells = case["n"] ** 3
    return {"bytes": 16 * N * cells * case["nsteps"], "flops": 3 * f * cells * case["nsteps"]}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind not in ("step", "host", "rhs"):
        return None  # adaptive integrator, hierarchy of boxes, gradient through many steps
    P = _params(case)
    n = _cells3(case)
    g = _geom(case["flow"], n)
    dx = [g.dx[d] for d in range(3)]
    if kind == "rhs":
        S = _flow(case, P, [q + 2 * G for q in n], seed)
        ds, fl = _x_rhs(P, S, dx)
        return {"dsdt": list(ds.unbind(0)), "flux": fl}
    S0 = _flow(case, P, n, seed)
    dt = _x_timestep(P, S0, dx)
    per = [bool(g.is_periodic[d]) for d in range(3)]
    boxes = chop((0, 0, 0), [q - 1 for q in n], case["max_grid"])
    S, norms = _x_step(P, S0, dx, per, dt, boxes)
    flat = torch.cat([S[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1].reshape(-1) for lo, hi in boxes])
    out = {"state": flat, "norms": norms}
    if kind == "step":
        out["dt"] = np.array([dt])
    return out


def _x_timestep(P, S, dx):
    vf = S[VFRAC]
    spec = S[NF:]
    ss = torch.sqrt(_thermo_gamma(P, S[DENS], spec) * S[PRES] / S[DENS])
    sp = torch.sqrt(S[VELX] ** 2 + S[VELX + 1] ** 2 + S[VELX + 2] ** 2)
    ws = float(torch.where(vf > 0, sp + ss, torch.zeros_like(sp)).max())
    md = 0.0
    for s in range(P.nspec):
        d = P.diff_gas[s] * vf + P.diff_solid[s] * (1 - vf) if P.diff_mode[s] else P.diff_gas[s] * torch.ones_like(vf)
        md = max(md, float(d.max()))
    dt = min(q / ws for q in dx) if ws > 0 else 1.7976931348623157e308
    if md > 0:
        dt = min([dt] + [0.5 * q * q / md / 3 for q in dx])
    return dt * P.cfl


def _x_faces(A, d, q=0, t=None, tq=0):
    """Cells of a grown array at offset q along d (and tq along t) from the
    right cell of every face of direction d."""
    sl = [slice(None)] * (A.dim() - 3)
    for e in (2, 1, 0):
        n = A.shape[-1 - e] - 2 * G
        o = G + (q if e == d else 0) + (tq if e == t else 0)
        sl.append(slice(o, o + n + (1 if e == d else 0)))
    return A[tuple(sl)]


def _x_valid(A):
    return A[..., G:-G, G:-G, G:-G]


def _x_weno(a, b, c, d, e):
    b2 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b0 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    w2, w1, w0 = 0.1 / (1e-6 + b2) ** 2, 0.6 / (1e-6 + b1) ** 2, 0.3 / (1e-6 + b0) ** 2
    num = w2 * (2 * a - 7 * b + 11 * c) + w1 * (-b + 5 * c + 2 * d) + w0 * (2 * c + 5 * d - e)
    return num / (6 * (w2 + w1 + w0))


def _x_limited(um, ul, ur, up):
    d1, d2 = up - ur, ul - um
    q = (d1 - d2).abs() / (d1.abs() + d2.abs() + 1e-20)
    h = 0.25 * (1 - q * q) * (d1 + d2)
    return ul + h, ur - h


def _x_hmean(a, b):
    return 2 * a * b / (a + b + 1e-30)


def _x_blend(mode, gas, solid, vf):
    return gas * vf + solid * (1 - vf) if mode else gas * torch.ones_like(vf)


def _x_ausm(P, uL, uR, d):
    def side(u):
        r = u[0]
        ke = 0.5 * (u[1] ** 2 + u[2] ** 2 + u[3] ** 2) / r
        p = _thermo_p(P, u[4] - ke, r, u[5:])
        gam = _thermo_gamma(P, r, u[5:])
        v = u[1 + d] / r
        H = gam / (gam - 1) * p / r + ke / r
        a = torch.sqrt(2 * (gam - 1) / (gam + 1) * H)
        return r, p, v, a * a / torch.maximum(a, v.abs())

    rL, pL, vL, aL = side(uL)
    rR, pR, vR, aR = side(uR)
    ah = torch.minimum(aL, aR)
    ML, MR = vL / ah, vR / ah
    mb2 = 0.5 * (ML ** 2 + MR ** 2)
    mo = torch.sqrt(torch.clamp(mb2, min=0.09, max=1.0))
    fa = mo * (2 - mo)
    alpha = 3 / 16 * (-4 + 5 * fa * fa)

    def mach(M, s):
        sub = s * 0.25 * (M + s) ** 2 + s * 0.125 * (M * M - 1) ** 2
        return torch.where(M.abs() <= 1, sub, 0.5 * (M + s * M.abs()))

    def pres(M, s):
        sub = 0.25 * (M + s) ** 2 * (2 - s * M) + s * alpha * M * (M * M - 1) ** 2
        return torch.where(M.abs() <= 1, sub, 0.5 * (M + s * M.abs()) / torch.where(M == 0, torch.ones_like(M), M))

    Mh = mach(ML, 1.0) + mach(MR, -1.0)
    Mh = Mh - 0.25 / fa * torch.clamp(1 - mb2, min=0) * (pR - pL) / (0.5 * (rL + rR) * ah * ah)
    mod = torch.where(Mh.abs() <= 0.3, (Mh * Mh + 0.09) / 0.6, Mh.abs())
    PL, PR = pres(ML, 1.0), pres(MR, -1.0)
    ph = PL * pL + PR * pR - 0.75 * PL * PR * (rL + rR) * fa * ah * (vR - vL)
    fL, fR = uL.clone(), uR.clone()
    fL[4] += pL
    fR[4] += pR
    fh = (0.5 * Mh * (fL + fR) - 0.5 * mod * (fR - fL)) * ah
    fh[1 + d] += ph
    return fh


def _x_rhs(P, S, dx):
    """dsdt on the valid box and the face fluxes of a grown state."""
    ns, N = P.nspec, NF + P.nspec
    comp = list(range(5)) + list(range(NF, N))
    order = P.order_hyp
    rho = S[RHO]
    vel = [S[RHOU + a] / rho for a in range(3)]
    ke2 = vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2
    spec = S[NF:]
    fluxes = []
    ds = torch.zeros((N,) + tuple(_x_valid(rho).shape), dtype=S.dtype, device=S.device)
    if order >= 4:
        p = _thermo_p(P, S[RHOE] - 0.5 * rho * ke2, rho, spec)
        reig = S[RHOE] - 0.5 * (S[1] ** 2 + S[2] ** 2 + S[3] ** 2) / rho
        gam = _thermo_gamma(P, rho, spec)
    for d in range(3):
        t1, t2 = (d + 1) % 3, (d + 2) % 3
        at = lambda A, q=0, t=None, tq=0: _x_faces(A, d, q, t, tq)  # noqa: E731
        vf = S[VFRAC]
        active = 0.5 * (at(vf, -1) + at(vf)) >= 0.5
        fall = at(vf, -3) < 1
        for q in range(-2, 3):
            fall = fall | (at(vf, q) < 1)
        mean = lambda A, t=None, tq=0: 0.5 * (at(A, -1, t, tq) + at(A, 0, t, tq))  # noqa: E731
        F = torch.zeros((N,) + tuple(active.shape), dtype=S.dtype, device=S.device)
        if order >= 4:
            aL = torch.sqrt(at(gam, -1) * _thermo_p(P, at(reig, -1), at(rho, -1), at(spec, -1)) / at(rho, -1))
            sR = at(spec, -1) if order == 5 else at(spec)
            aR = torch.sqrt(at(gam) * _thermo_p(P, at(reig), at(rho), sR) / at(rho))
            lam = torch.maximum(aL, aR) + torch.maximum(at(vel[d], -1).abs(), at(vel[d]).abs())
            for c in comp:
                u = S[c]
                f = u * vel[d] if c != RHOE else (u + p) * vel[d]
                if c == 1 + d:
                    f = f + p
                ul, ur, fl, fr = at(u, -1), at(u), at(f, -1), at(f)
                us = [torch.where(fall, ul if q < 0 else ur, at(u, q)) for q in range(-3, 3)]
                fs = [torch.where(fall, fl if q < 0 else fr, at(f, q)) for q in range(-3, 3)]
                if order == 5:
                    h = 0.5 * (_x_weno(*fs[:5]) + lam * _x_weno(*us[:5])) \
                        + 0.5 * (_x_weno(*fs[:0:-1]) - lam * _x_weno(*us[:0:-1]))
                else:
                    k = 0.08333333333
                    h = k * (7 * fs[3] + 7 * fs[2] - fs[1] - fs[4]) \
                        - k * (3 * us[3] - 3 * us[2] - us[4] + us[3]) * lam * P.dissfactor
                F[c] = h
        else:
            both = []
            for c in comp:
                ul, ur = at(S[c], -1), at(S[c])
                if order == 2:
                    um, up = torch.where(fall, ul, at(S[c], -2)), torch.where(fall, ur, at(S[c], 1))
                    ul, ur = _x_limited(um, ul, ur, up)
                both.append((ul, ur))
            fh = _x_ausm(P, torch.stack([b[0] for b in both]), torch.stack([b[1] for b in both]), d)
            del both
            for i, c in enumerate(comp):
                F[c] = fh[i]
            del fh
        for s in range(ns):
            F[NF + s] *= P.advect_flag[s]
        V = [S[VELX + a] for a in range(3)]
        gn = [(at(V[a]) - at(V[a], -1)) / dx[d] for a in range(3)]
        gt = lambda A, t: (mean(A, t, 1) - mean(A, t, -1)) / (2 * dx[t])  # noqa: E731
        mu = _x_hmean(P.visc_gas, P.visc_gas)
        div = gn[d] + gt(V[t1], t1) + gt(V[t2], t2)
        wk = 0.0
        for a in range(3):
            tau = mu * (2 * gn[d] - 2 / 3 * div) if a == d else mu * (gn[a] + gt(V[d], a))
            F[1 + a] -= tau
            wk = wk + tau * mean(V[a])
        F[RHOE] -= wk
        F *= active
        F[RHOE] -= _x_hmean(P.cond_gas, P.cond_gas) * (at(S[TEMP]) - at(S[TEMP], -1)) / dx[d]
        for s in range(ns):
            D = _x_hmean(_x_blend(P.diff_mode[s], P.diff_gas[s], P.diff_solid[s], at(vf, -1)),
                         _x_blend(P.diff_mode[s], P.diff_gas[s], P.diff_solid[s], at(vf)))
            F[NF + s] -= D * (at(S[NF + s]) - at(S[NF + s], -1)) / dx[d]
        m = F.shape[-1 - d] - 1
        ds += (F.narrow(3 - d, 0, m) - F.narrow(3 - d, 1, m)) / dx[d]
        fluxes.append(F)
    keep = _x_valid(S[VFRAC]) >= 1
    nmask = NF if P.species_in_solid == 1 else N
    ds[:nmask] *= keep
    ds += 0.0
    return ds, fluxes


def _x_external(P, E, d, s):
    """Ghost state of an ext_dir face from the boundary cells s (ncomp, ...)."""
    ones = torch.ones_like(s[DENS])
    spec = [E.spec[q] * ones for q in range(P.nspec)]
    if E.kind == abi.EXT_PRESSURE_INLET:
        vel = [0 * ones] * 3
        vel[d] = torch.sqrt(s[VELX] ** 2 + s[VELX + 1] ** 2 + s[VELX + 2] ** 2)
        rho, p = E.dens * ones, E.pres * ones
    elif E.kind == abi.EXT_PRESSURE_OUTLET:
        rho, p, vel, spec = s[DENS], E.pres * ones, [s[VELX + a] for a in range(3)], list(s[NF:])
    else:
        rho, p, vel = E.dens * ones, E.pres * ones, [E.vel[a] * ones for a in range(3)]
    return _from_prim(P, rho, vel, p, spec, s[VFRAC])


def _x_fill(P, S, per):
    n = [S.shape[-1 - d] for d in range(3)]
    B = torch.zeros((S.shape[0],) + tuple(n[e] + 2 * G for e in (2, 1, 0)), dtype=S.dtype, device=S.device)
    idx = []
    for d in range(3):
        i = torch.arange(-G, n[d] + G, device=S.device)
        idx.append(i % n[d] if per[d] else i.clamp(0, n[d] - 1))
    B.copy_(S[:, idx[2]][:, :, idx[1]][:, :, :, idx[0]])
    for stage in (1, 2, 3):
        for code in range(27):
            out = [(code // 3 ** d) % 3 - 1 for d in range(3)]
            if any(o and per[d] for d, o in enumerate(out)) or sum(map(abs, out)) != stage:
                continue
            ext = [d for d in range(3) if out[d] and (P.bc_lo[d] if out[d] < 0 else P.bc_hi[d]) == abi.BC_EXT_DIR]
            ds = ext[-1] if ext else [d for d in range(3) if out[d]][-1]
            kind = P.bc_lo[ds] if out[ds] < 0 else P.bc_hi[ds]
            dst, src = [slice(None)], [slice(None)]
            flip = False
            for d in (2, 1, 0):
                r = {-1: slice(0, G), 1: slice(n[d] + G, n[d] + 2 * G),
                     0: slice(0, n[d] + 2 * G) if per[d] else slice(G, n[d] + G)}[out[d]]
                dst.append(r)
                if d != ds:
                    src.append(r)
                elif kind == abi.BC_WALL:
                    src.append(slice(G, 2 * G) if out[d] < 0 else slice(n[d], n[d] + G))
                    flip = True
                else:
                    src.append(slice(G, G + 1) if out[d] < 0 else slice(n[d] + G - 1, n[d] + G))
            v = B[tuple(src)]
            if flip:
                v = torch.flip(v, [3 - ds]).clone()
                for c in (1, 2, 3, VELX, VELX + 1, VELX + 2):
                    v[c] = -v[c]
            elif kind == abi.BC_EXT_DIR:
                v = _x_external(P, P.ext_lo[ds] if out[ds] < 0 else P.ext_hi[ds], ds, v)
            B[tuple(dst)] = v.expand(B[tuple(dst)].shape)
    return B


def _x_cutcells(P, B, dx):
    vf = B[VFRAC]
    cut = torch.zeros_like(vf, dtype=torch.bool)
    v = _x_valid(vf)
    _x_valid(cut).copy_((v > 0) & (v < 1))
    o = cut.reshape(-1).nonzero().squeeze(1)
    if o.numel() == 0:
        return
    nx, ny = vf.shape[2], vf.shape[1]
    step = [1, nx, nx * ny]
    flat = [B[c].reshape(-1) for c in range(B.shape[0])]
    V = flat[VFRAC]
    dm = min(dx)
    gr = [(V[o + step[d]] - V[o - step[d]]) * (0.5 / dx[d]) for d in range(3)]
    mag = torch.sqrt(gr[0] ** 2 + gr[1] ** 2 + gr[2] ** 2)
    ok = mag > 1e-20
    sm = torch.where(ok, mag, torch.ones_like(mag))
    dist = torch.where(ok, (V[o] - 0.5) / sm, torch.zeros_like(mag))
    xp = [torch.where(ok, -dist * gr[d] / sm, torch.zeros_like(mag)) / dm for d in range(3)]
    names = [VELX, VELX + 1, VELX + 2, PRES, TEMP, DENS] + ([] if P.species_in_solid else list(range(NF, B.shape[0])))
    acc = {c: torch.zeros_like(mag) for c in names}
    swd, swn = torch.zeros_like(mag), torch.zeros_like(mag)
    for l3 in range(125):
        off = [l3 % 5 - 2, (l3 // 5) % 5 - 2, l3 // 25 - 2]
        q = o + sum(off[d] * step[d] for d in range(3))
        m = (V[q] == 1.0).to(V.dtype)
        r = [off[d] * dx[d] / dm for d in range(3)]
        wn = m / (sum((r[d] - xp[d]) ** 2 for d in range(3)) + 1e-40)
        wd = m * (0.0 if off == [0, 0, 0] else 1.0 / sum(x * x for x in r))
        swd += wd
        swn += wn
        for c in names:
            acc[c] += flat[c][q] * (wd if VELX <= c <= VELX + 2 else wn)
    have = swn > 0
    sw = torch.where(have, swn, torch.ones_like(swn))
    near = dist.abs() < dm * 1e-5
    dn = torch.where(near, torch.ones_like(dist), dist.abs() / dm)
    iden = torch.where(near, torch.zeros_like(dist), 1.0 / (swd + 1.0 / (dn * dn)))
    val = {c: (acc[c] * iden if VELX <= c <= VELX + 2 else torch.where(have, acc[c] / sw, flat[c][o])) for c in names}
    vel = [val[VELX + a] for a in range(3)]
    spec = [val.get(NF + s, flat[NF + s][o]) for s in range(P.nspec)]
    new = _from_prim(P, val[DENS], vel, val[PRES], spec, V[o])
    new[TEMP] = val[TEMP]
    for c in range(B.shape[0]):
        flat[c][o] = new[c]


def _x_chem(P, s0, T, dt):
    if not P.chem_on:
        return s0.clone()
    kr = [P.A[r] * torch.exp(-P.Ea[r] / (cases.RU * T)) if P.Ea[r] else P.A[r] * torch.ones_like(T)
          for r in range(P.nreact)]

    def source(s):
        w = torch.zeros_like(s)
        for r in range(P.nreact):
            rate = kr[r]
            for q in range(P.nspec):
                if P.order[r][q] > 0:
                    rate = rate * s[q] ** P.order[r][q]
            for q in range(P.nspec):
                if P.nu[r][q]:
                    w[q] += P.nu[r][q] * rate
        return w

    f0 = source(s0)
    f1 = source(s0 + dt * f0)
    f2 = source(s0 + 0.25 * dt * (f0 + f1))
    return s0 + dt * (f0 / 6 + f1 / 6 + 2 / 3 * f2)


def _x_step(P, S0, dx, per, dt, boxes):
    third = 0.6666666666666666667 * 0.5
    S = S0
    for stage in (1, 2, 3):
        filled = _x_fill(P, S, per)
        T = torch.empty_like(S)
        for lo, hi in boxes:  # a box's ghost cells keep their filled values: the cut cells are its valid ones
            at = (slice(None),) + tuple(slice(lo[e], hi[e] + 1) for e in (2, 1, 0))
            B = filled[(slice(None),) + tuple(slice(lo[e], hi[e] + 1 + 2 * G) for e in (2, 1, 0))].clone()
            _x_cutcells(P, B, dx)
            ds = _x_rhs(P, B, dx)[0]
            if stage == 1:
                T[at] = _x_valid(B) + dt * ds
            elif stage == 2:
                T[at] = ((S[at] + dt * ds) + 3.0 * S0[at]) * 0.25
            else:
                T[at] = (S0[at] + 2.0 * (S[at] + dt * ds)) * third
        S = T
    old = S
    S = S.clone()
    S[NF:] = _x_chem(P, old[NF:], old[TEMP], dt)
    gas = S[VFRAC] == 1.0
    rho = S[RHO]
    vel = [S[RHOU + a] / rho for a in range(3)]
    p = _thermo_p(P, S[RHOE] - 0.5 * rho * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2), rho, S[NF:])
    for c, v in ((DENS, rho), (VELX, vel[0]), (VELX + 1, vel[1]), (VELX + 2, vel[2]), (PRES, p),
                 (TEMP, _thermo_t(P, rho, p, S[NF:]))):
        S[c] = torch.where(gas, v, S[c])
    S[NF:].clamp_(min=0.0)
    r = (S - old) / dt
    r[:VFRAC] *= old[VFRAC]
    return S, r.reshape(r.shape[0], -1).square().sum(1).sqrt().cpu().numpy()
