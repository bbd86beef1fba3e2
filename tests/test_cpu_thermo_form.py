"""The thermodynamics the kernels use in place of the plugins' expressions
(thermo.H get_p_from_rec, get_gama_from_rc; flux_schemes.H:21-43), in plain
float64 against the plugins' formulas in extended precision: kappa = R sum(c)
/ sum(cv c) is gamma - 1 and p / (rho e), total enthalpy is (E + p) / rho, and
the AUSM+-up factor 2 (gamma - 1) / (gamma + 1) is 2 n / (2 d + n).  Each is a
chain of fewer than 12 roundings of positive quantities: 12 eps relative."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps
L = np.longdouble
R = 8.31446261815324


@pytest.mark.parametrize("ns", [1, 2, 5, 8])
def test_kappa_pressure_gamma_enthalpy(ns):
    rng = np.random.default_rng(ns)
    n = 100000
    gam = rng.uniform(1.1, 1.67, ns)
    c = rng.gamma(1.0, 1.0, (ns, n)) * 10.0 + 1e-12
    rhoe = 10.0 ** rng.uniform(3, 7, n)
    cv = R / (gam - 1.0)
    sums, cvs = np.zeros((2, n)), np.zeros((2, n))
    for s in range(ns):
        sums[s & 1] += c[s]
        cvs[s & 1] += cv[s] * c[s]
    num, den = R * (sums[0] + sums[1]), cvs[0] + cvs[1]
    kap = num / den
    T = L(1) * rhoe / sum(L(R) / (L(gam[s]) - 1) * c[s] for s in range(ns))
    p_ref = sum(L(R) * c[s] * T for s in range(ns))
    tot = sum(L(1) * c[s] for s in range(ns))
    gam_ref = 1 + 1 / sum((c[s] / tot) / (L(gam[s]) - 1) for s in range(ns))
    assert np.all(np.abs(kap * rhoe - p_ref) <= 12 * EPS * p_ref)
    assert np.all(np.abs((1.0 + kap) - gam_ref) <= 12 * EPS * gam_ref)
    assert np.all(np.abs(num * (rhoe / den) - p_ref) <= 12 * EPS * p_ref)
    af_ref = 2 * (gam_ref - 1) / (gam_ref + 1)
    assert np.all(np.abs((2.0 * num) / (2.0 * den + num) - af_ref) <= 12 * EPS * af_ref)
    # gamma/(gamma-1) p/rho + k = (E + p)/rho with E = rho e + rho k
    rho, k = 10.0 ** rng.uniform(-1, 1, n), 10.0 ** rng.uniform(-3, 5, n)
    E = rhoe + rho * k
    h_ref = gam_ref / (gam_ref - 1) * p_ref / rho + k
    assert np.all(np.abs((E + kap * rhoe) / rho - h_ref) <= 12 * EPS * h_ref)
