"""The order-5 flux beside a front (mfg_weno_weights.cuh, compiled here for the
host): second differences with fixed-point weights, or, where weno_front says
so, the weighted candidates, against the candidate form in extended precision.

Bounds, derived beforehand, relative to the values at the face and the parts of
the flux (weights times absolute candidates).  Candidates: an indicator within 5
roundings, a weight 12, a candidate 3, sum, reciprocal and product 8: below 64
eps for the four edges.  Elsewhere the largest difference is below 2^8 of the
face's values (E <= S + 7 in exponents), and the sum's three roundings are of
quantities below 8 differences over 12: 2^8 x 2 eps."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EPS = np.finfo(np.float64).eps
L = np.longdouble
N = 20000

SHIM = r"""
#include <math.h>
#include <string.h>
#include "mfg_weno_weights.cuh"
using namespace mfg;
static double val(uint64_t u) { return double_of(u); }
static double correction(const double* v, bool state, int& top) {
    double d[5], t[4];
    for (int q = 0; q < 5; ++q) d[q] = v[q + 1] - v[q];
    for (int q = 0; q < 4; ++q) t[q] = d[q + 1] - d[q];
    WenoInd c[4];
    for (int q = 0; q < 4; ++q) c[q] = weno_ind(weno_diff(bits_of(d[q])), weno_diff(bits_of(d[q + 1])));
    top = imax(imax(c[0].eB, c[1].eB), imax(c[2].eB, c[3].eB));
    const WenoWeights l = weno_weights(c[0].dB, c[0].eB, c[1].dC, c[1].eC, c[2].dA, c[2].eA);
    const WenoWeights r = weno_weights(c[1].dB, c[1].eB, c[2].dC, c[2].eC, c[3].dA, c[3].eA);
    const double g0 = t[1] - t[0], g1 = t[2] - t[1], g2 = t[3] - t[2];
    if (state)
        return fma(val(r.farR2), g2, fma(val(signed_weight_bits((l.qL + r.qR) - ((int64_t)1 << 62))), g1, val(l.farL2) * g0));
    return fma(-val(r.farR2), g2, fma(val(signed_weight_bits(l.qL - r.qR)), g1, fma(val(l.farL2), g0, t[1]) + t[2]));
}
// f, u: six cells per face; pressure: the flux is a momentum's along the face normal; out: the flux; front: whether the candidates gave it
extern "C" void flux(const double* f, const double* u, const double* lam, double* out, int* front, int pressure, int n) {
    for (int i = 0; i < n; ++i, f += 6, u += 6) {
        int tf, tu;
        const double C = correction(f, false, tf), U = correction(u, true, tu);
        front[i] = weno_front(tf, tu, pressure, f[2], f[3], u[2], u[3], lam[i]);
        if (front[i]) {
            const double fp = weno_front_edge(f[0], f[1], f[2], f[3], f[4]), fm = weno_front_edge(f[5], f[4], f[3], f[2], f[1]);
            const double up = weno_front_edge(u[0], u[1], u[2], u[3], u[4]), um = weno_front_edge(u[5], u[4], u[3], u[2], u[1]);
            out[i] = (fma(lam[i], up, fp) + fma(-lam[i], um, fm)) / 12;
        } else {
            out[i] = 0.5 * fma(-1.0 / 6.0, fma(lam[i], U, C), f[2] + f[3]);
        }
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("front")
    src, so = str(d / "w.cpp"), str(d / "w.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mesoflow_gb300", "csrc"), src, "-o", so],
                   check=True, capture_output=True)
    return C.CDLL(so)


def flux(lib, f, u, lam, pressure=False):
    f, u = (np.ascontiguousarray(x.T) for x in (f, u))
    out, front = np.empty(lam.size), np.empty(lam.size, np.int32)
    lib.flux(*[x.ctypes.data_as(C.c_void_p) for x in (f, u, lam, out, front)], C.c_int(int(pressure)), C.c_int(lam.size))
    return out, front


def edge(a, b, c, d, e, absolute):
    k, eps = L(13) / L(12), L(1e-6)
    w = [1 / (eps + k * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4) ** 2,
         6 / (eps + k * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4) ** 2,
         3 / (eps + k * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4) ** 2]
    if absolute:
        a, b, c, d, e = (np.abs(x) * q for x, q in ((a, 1), (b, -1), (c, 1), (d, 1), (e, -1)))
        v = [2 * a - 7 * b + 11 * c, -b + 5 * c + 2 * d, 2 * c + 5 * d - e]
    else:
        v = [2 * a - 7 * b + 11 * c, -b + 5 * c + 2 * d, 2 * c + 5 * d - e]
    return sum(p * q for p, q in zip(w, v)) / (6 * sum(w))


def check(lib, f, u, lam, pressure=False):
    got, front = flux(lib, f, u, lam, pressure)
    F, U, l = [L(x) for x in f], [L(x) for x in u], L(lam)
    want = (edge(*F[:5], False) + l * edge(*U[:5], False) + edge(*F[:0:-1], False) - l * edge(*U[:0:-1], False)) / 2
    part = edge(*F[:5], True) + l * edge(*U[:5], True) + edge(*F[:0:-1], True) + l * edge(*U[:0:-1], True)
    here = np.maximum(np.maximum(np.abs(f[2]), np.abs(f[3])), lam * np.maximum(np.abs(u[2]), np.abs(u[3])))
    err = np.abs(got - want).astype(float)
    bound = EPS * np.where(front, 64 * part.astype(float), 64 * part.astype(float) + 512 * here)
    assert np.all(err <= bound), np.max(err / bound)
    return front


@pytest.mark.parametrize("low,high", [(1e-9, 1.0), (0.0, 50.0), (1e-12, 50.0), (1e-9, 1e3), (0.0, 1e3), (1e-3, 1.0),
                                      (1e-300, 1e5), (1e-2, 1.0), (0.1, 1.0), (1.0, 1e5), (1e5, 1e17)])
@pytest.mark.parametrize("at", [1, 2, 3, 4, 5])
def test_front(lib, low, high, at):
    rng = np.random.default_rng(at)
    for left in (False, True):
        side = (np.arange(6) < at) == left
        u = np.where(side[:, None], high, low) * (1 + 0.01 * rng.standard_normal((6, N)))
        f = u * (5 * rng.standard_normal(N) + 0.1 * rng.standard_normal((6, N)))
        front = check(lib, f, u, 335 + 10 * rng.random(N))
        if low <= 1e-3 * high and at in (1, 2, 4, 5) and (at < 3) == left:  # low beside the face
            assert np.all(front)


def test_any_ratio(lib):
    """Ratios about the rule's line, jumps about the exponent floor, and values
    of every size."""
    rng = np.random.default_rng(2)
    side = np.arange(6)[:, None] < rng.integers(0, 7, N)
    for low, high in ((10.0 ** rng.uniform(-6, 0, N), 2.0 ** rng.uniform(3, 10, N)),
                      (1e-4 * rng.random(N), 10.0 ** rng.uniform(0, 4, N)),
                      (10.0 ** rng.uniform(-12, 8, N), 10.0 ** rng.uniform(0, 14, N))):
        u = np.where(side, low * high, low) * (1 + 0.1 * rng.standard_normal((6, N)))
        lam = 10.0 ** rng.uniform(-2, 4, N)
        check(lib, u * lam * (0.3 * rng.standard_normal(N) + 0.05 * rng.standard_normal((6, N))), u, lam)


def test_smooth_data_keeps_the_fixed_point_form(lib):
    """A sine through zero with ten cells per half wave, its flux and its square:
    no face is a front."""
    x = 2 * np.pi * np.random.default_rng(4).random(N) + 0.3 * np.arange(6)[:, None]
    u = 30 * np.sin(x)
    for f in (u * 20 * np.cos(x + 1), u * u / 1.2 + 1e5):
        assert not np.any(check(lib, f, u, np.full(N, 400.0), pressure=f.min() > 0))


def test_momentum_beside_a_pressure_jump(lib):
    """The momentum along the normal: its flux holds the pressure, on the low side
    of a jump of it far below the other side's and far above lam |u|."""
    rng = np.random.default_rng(9)
    side = np.arange(6)[:, None] < rng.integers(0, 7, N)
    u = rng.choice([0.0, 1e-6, 1.0], N) * rng.standard_normal((6, N))
    p = np.where(side, 1.0, 10.0 ** rng.uniform(0, 6, N)) * 1e4 * (1 + 0.01 * rng.standard_normal((6, N)))
    check(lib, u * u / 1.2 + p, u, np.full(N, 350.0), pressure=True)


def test_infinite_cells_take_the_candidates(lib):
    """An infinite or NaN cell in the stencil gives a NaN flux, as the candidate
    form's, never a finite or an infinite one."""
    for bad in (np.inf, -np.inf, np.nan):
        for q in range(6):
            u = 1.0 + 0.1 * np.random.default_rng(q).random((6, 8))
            f = 3.0 * u
            for v in (u, f):
                w = v.copy()
                w[q] = bad
                out, front = flux(lib, *((w, u) if v is f else (f, w)), np.full(8, 2.0))
                assert np.all(front) and np.all(np.isnan(out))
