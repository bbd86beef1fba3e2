"""The reversed fluxes beside a front: the gradient with respect to the inlet
velocity of the reaction rate of a trace species, two cells from a front to a
value many orders of magnitude above it.  The column sweep against the per-face
form (FP64 candidates throughout), whose sums run in another order: each of the
few hundred terms rounds to within a few eps, and none is larger than the result
by more than ten: 1e-12."""
import math

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.adjoint import ReactionProblem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def problem(low, high, n=16):
    """gas 1 + site 8 -> gas 2 + site 9 in the cells at the inlet; gas 1 is low in
    two cells, high from the third on.  The step is so short that the front does
    not move, and nothing diffuses."""
    c = cases.catalyst(n=n, order=5, max_grid=8)
    P = c.params
    P.nreact = 1
    for s in range(abi.MAX_SPECIES):
        P.nu[0][s] = P.order[0][s] = P.diff_gas[s] = P.diff_solid[s] = 0.0
    for s, v in ((1, -1.0), (8, -1.0), (2, 1.0), (9, 1.0)):
        P.nu[0][s] = v
    P.order[0][1] = P.order[0][8] = 1.0
    P.A[0], P.Ea[0] = 1e2, 0.0
    rng = np.random.default_rng(3)
    shape = c.state.shape[1:]
    x = np.indices(shape)[2]
    noise = lambda a: 1.0 + a * rng.standard_normal(shape)
    spec = [24.0 * noise(0.01), np.where(x < 2, low, high) * noise(0.01)] + [0.1 * noise(0.01) for _ in range(6)]
    spec += [np.where(x < 1, 3.0, 0.0), np.where(x < 1, 1.0, 0.0)]
    rho = sum(spec[s] * P.molwt[s] for s in range(8))
    vel = [v * noise(0.05) for v in (0.5, 0.1, 0.1)]
    c.state = cases.state_from_prim(P, rho, *vel, 1e5 * noise(0.001), spec, np.ones(shape))
    e = P.ext_lo[0]
    e.dens = float(rho[:, :, 0].mean())
    for s in range(8):
        e.spec[s] = float(spec[s][:, :, 0].mean())
    return ReactionProblem(c, 1, 2e-16, checkpoint_every=0), np.array([math.log(P.A[0])])


@pytest.mark.parametrize("low,high", [(1e-9, 8.0), (1e-6, 8.0), (1e-10, 0.5), (1.0, 8.0)])
def test_trace_gradient(low, high):
    p, log_a = problem(low, high)
    lib = abi.load()
    out = []
    for form in (0, 1):
        abi.check("form", lib.mfg_set_adjoint_flux_form(form))
        try:
            out.append(p.gradient(log_a, 1.0))
        finally:
            abi.check("form", lib.mfg_set_adjoint_flux_form(1))
    (j0, a0, u0), (j1, a1, u1) = out
    print(low, high, "dJ/du_in", u0, u1, abs(u1 / u0 - 1.0))
    assert abs(j1 - j0) <= 1e-13 * abs(j0)
    assert abs(a1[0] - a0[0]) <= 1e-12 * abs(a0[0])
    assert u0 != 0.0 and abs(u1 - u0) <= 1e-12 * abs(u0)
