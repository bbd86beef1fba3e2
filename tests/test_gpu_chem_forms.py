"""Chemistry sub-steps where their short cuts begin and end: cells without a
reactant (no exponential is evaluated for them), temperatures and constants
for which that is not allowed, reaction orders beside 1 and 2, at every species
count the kernels are built for, and the implicit form with its rate constants
evaluated once."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _case(nspec, nreact, seed, n=(7, 5, 6)):
    """A reaction table over nspec species: orders 1, 2, 1.5 and 2.5,
    constants with and without an activation energy."""
    rng = np.random.default_rng(seed)
    c = cases.catalyst(n=8, order=5, max_grid=8)
    P = c.params
    P.nspec = P.ngas = nspec
    P.nreact = nreact
    for r in range(abi.MAX_REACTIONS):
        for s in range(abi.MAX_SPECIES):
            P.nu[r][s] = P.order[r][s] = 0.0
    for s in range(nspec):
        P.molwt[s], P.gamma[s] = 0.02 + 0.001 * s, 1.3
    for r in range(nreact):
        a, b = (rng.choice(nspec, size=2, replace=False) if nspec > 1 else (0, 0))
        P.nu[r][a] -= 1.0
        P.nu[r][b] += 0.5
        P.order[r][a] = (1.0, 2.0, 1.5, 2.5)[r % 4]
        if nspec > 1 and r % 3 == 0:
            P.order[r][b] = 1.0
        P.A[r] = 10.0 ** rng.uniform(2.0, 4.0)
        P.Ea[r] = (0.0, 40e3, 90e3)[r % 3]
    y = rng.uniform(0.1, 2.0, size=(nspec,) + n[::-1])
    y[rng.uniform(size=y.shape) < 0.4] = 0.0
    T = rng.uniform(300.0, 900.0, size=n[::-1])
    return c, y, T


def _run(P, y, T, dt, kind, rtol=1e-6, atol=1e-12, boxes=1):
    lib = abi.load()
    abi.check("init", lib.mfg_init(C.byref(P)))
    abi.check("integrator", lib.mfg_set_chem_integrator(kind, rtol, atol, 5000))
    try:
        ns = y.shape[0]
        S = np.ones((abi.FLO_NVARS + ns,) + y.shape[1:])
        S[abi.FLO_NVARS:] = y
        S[abi.TEMP] = T
        hi = tuple(m - 1 for m in y.shape[:0:-1])
        lev = Level([((0, 0, 0), hi)] * boxes, S.shape[0], backend="torch", device="cuda")
        for t in lev.s_old:
            t.copy_(torch.as_tensor(S))
        geom = cases.catalyst(n=8).geom
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        abi.check("chem", lib.mfg_chem_substep(lev.descriptors(), boxes, C.byref(geom), 0.0, dt, st))
        torch.cuda.synchronize()
        out = [t.cpu().numpy() for t in lev.s_new]
        for o in out[1:]:
            assert np.array_equal(o, out[0], equal_nan=True)
        return out[0]
    finally:
        abi.check("integrator", lib.mfg_set_chem_integrator(0, 1e-8, 1e-12, 1000))


def _explicit(P, y, T, dt):
    """SSP-RK3 of the source in plain FP64 and the magnitude its terms have."""
    ns = y.shape[0]
    mag = np.abs(y).copy()
    with np.errstate(all="ignore"):
        kr = [P.A[r] * np.exp(-P.Ea[r] / (cases.RU * T)) if P.Ea[r] else P.A[r] * np.ones_like(T)
              for r in range(P.nreact)]

        def f(s):
            w = np.zeros_like(s)
            for r in range(P.nreact):
                cm = np.ones_like(T)
                for q in range(ns):
                    if P.order[r][q] > 0:
                        cm = cm * s[q] ** P.order[r][q]
                for q in range(ns):
                    if P.nu[r][q]:
                        w[q] += P.nu[r][q] * (kr[r] * cm)
                        mag[q] += np.abs(dt * P.nu[r][q] * kr[r] * cm)
            return w

        f0 = f(y)
        f1 = f(y + dt * f0)
        f2 = f((y + dt * 0.25 * f0) + dt * 0.25 * f1)
        return ((y + dt / 6 * f0) + dt / 6 * f1) + dt * (2.0 / 3.0) * f2, mag


@pytest.mark.parametrize("nspec", [1, 2, 4, 8, 9, 12, 13, 16])
def test_explicit_against_plain_form(nspec):
    """Difference bound, per component: the terms' magnitude (|y| and dt |nu|
    rate of the three stages) times the relative error of a rate: exp of an
    argument x = Ea/(RU T) < 40 known to 1.5 ulp (60 ulp), pow (2 ulp per
    factor), products and sums (10 ulp), carried into the later stages through
    a rate's sensitivity (factor 4 covers orders up to 2 twice)."""
    c, y, T = _case(nspec, min(3 * nspec, abi.MAX_REACTIONS), 11 + nspec)
    if nspec > 1:
        T.flat[:6] = (0.0, -0.0, np.inf, np.nan, 1e-310, 1e-3)  # zero rates, infinite ones and NaN
    dt = 1e-6
    got = _run(c.params, y, T, dt, 0)[abi.FLO_NVARS:]
    want, mag = _explicit(c.params, y, T, dt)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want) & np.isfinite(mag)
    assert ok.mean() > 0.9
    assert np.all(np.abs(got - want)[ok] <= 4 * 80 * 2 * EPS * mag[ok])


def test_explicit_untame_constants():
    """A negative activation energy, an infinite constant or a negative
    temperature makes the constant of a reaction without reactants infinite:
    0 x inf is NaN, as in the plain form."""
    c, y, T = _case(3, 3, 5)
    P = c.params
    P.Ea[0], P.Ea[1], P.A[2], P.Ea[2] = -60e3, 50e3, 1e300, 0.0
    T.flat[:4] = (1e-3, -1e-3, 500.0, -500.0)
    got = _run(P, y, T, 1e-9, 0)[abi.FLO_NVARS:]
    want, _ = _explicit(P, y, T, 1e-9)
    assert np.isnan(want[y == 0.0]).any()
    assert np.array_equal(np.isfinite(got), np.isfinite(want))


@pytest.mark.parametrize("nspec", [1, 3, 4, 5, 8, 9, 12, 13, 16])
def test_implicit_against_oracle(nspec):
    """Both sides take the same steps, so they differ by the Newton matrices'
    rounding: 16 rows, condition below 1e3 at h k <= 10, at most 80
    steps: 1e-9 of each cell's largest species is three decimals above it.
    Three boxes of 210 cells: the last block is not full."""
    c, y, T = _case(nspec, min(2 * nspec, abi.MAX_REACTIONS), 31 + nspec)
    P = c.params
    for r in range(P.nreact):  # integer orders, as the iteration passes through negative values
        for s in range(nspec):
            P.order[r][s] = 0.0 if P.order[r][s] == 0.0 else (2.0 if P.order[r][s] == 2.0 else 1.0)
    dt = 1e-4
    got = _run(P, y, T, dt, 1, rtol=1e-3, atol=1e-5, boxes=3)
    S = np.ones_like(got)
    S[abi.FLO_NVARS:], S[abi.TEMP] = y, T
    lev = Level([((0, 0, 0), tuple(m - 1 for m in y.shape[:0:-1]))], S.shape[0], backend="numpy")
    lev.s_old[0][...] = S
    lib = oracle_lib.load("strict")
    assert lib.oracle_chem_substep_ros2(C.byref(P), lev.descriptors(), 1, dt, 1e-3, 1e-5, 5000) == 0
    want = lev.s_new[0]
    sp = slice(abi.FLO_NVARS, None)
    scale = np.abs(want[sp]).max(axis=0, keepdims=True) + 1e-5
    assert np.max(np.abs(got[sp] - want[sp]) / scale) < 1e-9
    assert np.array_equal(got[:abi.FLO_NVARS], S[:abi.FLO_NVARS])
