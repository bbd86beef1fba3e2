"""The form of the WENO5 local Lax-Friedrichs flux that the order-5 kernels use
(second differences, weights in 64-bit fixed point from mfg_weno_weights.cuh,
compiled here for the host) against the reference's candidate form
(flux_schemes.H:373-495) in extended precision, on smooth, noisy,
discontinuous, constant, tiny, huge and collapsed (first-order fallback)
stencils.

Bounds, derived beforehand.  Weights: an indicator's fixed point truncates the
products D-^2, D- D+, D+^2 (coefficients up to 10, 11, 4, each by less than
one unit) of a sum that is at least 2^55 units, so its relative error is below
25 x 2^-55 < 2^-50; a weight is a ratio of products of two squared indicators,
w (1 - w) <= 1/4 times four such errors: 2^-50 absolute, plus the conversion's
2^-53.  Flux: every FP64 operation rounds to within half an ulp of a quantity
bounded by a small multiple of the scale s = max |f| + lam max |u| (a third
difference is at most 8 max |v|, taken over 12), and a weight's error moves
the flux by at most 2^-50 x 2 (8 + 8) / 12 s in the worst alignment; the
kernels' sum stays within 20 eps s."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EPS = np.finfo(np.float64).eps
L = np.longdouble
N = 50000

SHIM = r"""
#include <string.h>
#include "mfg_weno_weights.cuh"
using namespace mfg;
static uint64_t bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
static double val(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
// d: 4 differences per stencil; w: far and near weight of the left and of the right edge of its middle cell
extern "C" void weights(const double* d, double* w, int n) {
    for (int i = 0; i < n; ++i) {
        WenoInd c[3];
        for (int q = 0; q < 3; ++q) c[q] = weno_ind(weno_diff(bits(d[4 * i + q])), weno_diff(bits(d[4 * i + q + 1])));
        const WenoWeights r = weno_weights(c[0].dB, c[0].eB, c[1].dC, c[1].eC, c[2].dA, c[2].eA);
        w[4 * i] = 0.5 * val(r.farL2);
        w[4 * i + 1] = val(r.nearL);
        w[4 * i + 2] = 0.5 * val(r.farR2);
        w[4 * i + 3] = val(r.nearR);
    }
}
// weight W of the first-order stencil with the jump d, and D dW/dD over -4
extern "C" void collapsed(const double* d, double* w, double* q, int n) {
    for (int i = 0; i < n; ++i) {
        const WenoCollapsed c = weno_collapsed(weno_diff(bits(d[i])));
        w[i] = val(weight_bits(c.W, 0));
        q[i] = val(weno_collapsed_slope(c));
    }
}
// d: 5 differences per face; w: far weight of its left edge (twice), the near weights' sum less one and
// difference, far weight of its right edge (twice)
extern "C" void pairs(const double* d, double* w, int n) {
    for (int i = 0; i < n; ++i) {
        WenoInd c[4];
        for (int q = 0; q < 4; ++q) c[q] = weno_ind(weno_diff(bits(d[5 * i + q])), weno_diff(bits(d[5 * i + q + 1])));
        const WenoWeights l = weno_weights(c[0].dB, c[0].eB, c[1].dC, c[1].eC, c[2].dA, c[2].eA);
        const WenoWeights r = weno_weights(c[1].dB, c[1].eB, c[2].dC, c[2].eC, c[3].dA, c[3].eA);
        w[4 * i] = val(l.farL2);
        w[4 * i + 1] = val(signed_weight_bits((l.qL + r.qR) - ((int64_t)1 << 62)));
        w[4 * i + 2] = val(signed_weight_bits(l.qL - r.qR));
        w[4 * i + 3] = val(r.farR2);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("weno")
    src, so = str(d / "w.cpp"), str(d / "w.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mesoflow_gb300", "csrc"), src, "-o", so],
                   check=True, capture_output=True)
    return C.CDLL(so)


def fixed_weights(lib, d):
    d = np.ascontiguousarray(np.stack(d, axis=1))
    w = np.empty((d.shape[0], 4))
    lib.weights(d.ctypes.data_as(C.c_void_p), w.ctypes.data_as(C.c_void_p), C.c_int(d.shape[0]))
    return w.T


def edge_weights(a, b, c, d, g):
    k, e = L(13) / L(12), L(1e-6)
    q2 = (e + k * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4) ** 2
    q1 = (e + k * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4) ** 2
    q0 = (e + k * (c - 2 * d + g) ** 2 + (3 * c - 4 * d + g) ** 2 / 4) ** 2
    w2, w1, w0 = q1 * q0, 6 * q2 * q0, 3 * q2 * q1
    s = w2 + w1 + w0
    return w2 / s, w1 / s, w0 / s


def reference(f, u, lam):
    f, u, lam = [L(x) for x in f], [L(x) for x in u], L(lam)

    def edge(a, b, c, d, g):
        w2, w1, w0 = edge_weights(a, b, c, d, g)
        return (w2 * (2 * a - 7 * b + 11 * c) + w1 * (-b + 5 * c + 2 * d) + w0 * (2 * c + 5 * d - g)) / 6

    return (edge(*f[:5]) + lam * edge(*u[:5])) / 2 + (edge(*f[:0:-1]) - lam * edge(*u[:0:-1])) / 2


def kernel_form(lib, f, u, lam):
    def parts(v):
        d = [v[i + 1] - v[i] for i in range(5)]
        t = [d[i + 1] - d[i] for i in range(4)]
        g = [t[i + 1] - t[i] for i in range(3)]
        a = np.ascontiguousarray(np.stack(d, axis=1))
        w = np.empty((a.shape[0], 4))
        lib.pairs(a.ctypes.data_as(C.c_void_p), w.ctypes.data_as(C.c_void_p), C.c_int(a.shape[0]))
        return t, g, w.T

    t, g, w = parts(f)
    c = ((t[1] + w[0] * g[0]) + t[2]) + w[2] * g[1] - w[3] * g[2]  # sum of the two edges' corrections
    t, g, w = parts(u)
    d = w[0] * g[0] + w[1] * g[1] + w[3] * g[2]                     # difference of the state's
    return 0.5 * ((f[2] + f[3]) - (c + lam * d) / 6)


def collapsed_weight(lib, d):
    d = np.ascontiguousarray(d)
    w, q = np.empty_like(d), np.empty_like(d)
    p = [x.ctypes.data_as(C.c_void_p) for x in (d, w, q)]
    lib.collapsed(p[0], p[1], p[2], C.c_int(d.size))
    return w, q


def collapsed_form(lib, f, u, lam):
    d = u[3] - u[2]
    return 0.5 * ((f[2] + f[3]) - lam * d * collapsed_weight(lib, d)[0])


def stencils(kind, rng):
    if kind == "smooth":
        return 1e5 * (1.0 + 1e-4 * rng.standard_normal((6, N)))
    if kind == "noisy":
        return rng.gamma(2.0, 1.0, (6, N))
    if kind == "shock":
        return np.where(np.arange(6)[:, None] < rng.integers(0, 7, N), 1.0, 0.125) * (1 + 1e-3 * rng.standard_normal((6, N)))
    if kind == "large":
        return 10.0 ** rng.uniform(-3, 17, N) * rng.standard_normal((6, N))
    if kind == "tiny":
        return 10.0 ** rng.uniform(-300, -3, N) * rng.standard_normal((6, N))
    if kind == "constant":  # runs of equal cells, zeros of both signs among the differences
        return rng.choice([0.0, 1.0, -1.0, 3.5], size=(6, N))
    a, b = rng.standard_normal((2, N)) * 10.0 ** rng.uniform(-6, 6, N)  # collapsed
    return np.stack([a, a, a, b, b, b])


KINDS = ["smooth", "noisy", "shock", "large", "tiny", "constant", "collapsed"]


@pytest.mark.parametrize("kind", KINDS)
def test_fixed_point_weights(lib, kind):
    v = stencils(kind, np.random.default_rng(3))
    d = [v[i + 1] - v[i] for i in range(4)]
    w = fixed_weights(lib, d)
    x = [L(0) * L(d[0])]
    for q in d:  # the stencil whose differences are exactly d
        x.append(x[-1] + L(q))
    wl, wr = edge_weights(*x), edge_weights(*x[::-1])
    for got, ref in zip(w, (wl[0], wl[2], wr[0], wr[2])):
        assert np.all(np.abs(got - ref) <= 2.0 ** -50 + 2.0 ** -53)
        assert np.all(got >= 0.0) and np.all(got <= 1.0)


@pytest.mark.parametrize("kind", KINDS)
def test_flux_form(lib, kind):
    rng = np.random.default_rng(7)
    f, u = stencils(kind, rng), stencils(kind, rng)
    lam = rng.uniform(0.1, 10.0, N)
    ref = reference(f, u, lam)
    s = np.abs(f).max(0) + lam * np.abs(u).max(0)
    assert np.all(np.abs(kernel_form(lib, f, u, lam) - ref) <= 20 * EPS * s)
    if kind == "collapsed":
        assert np.all(np.abs(collapsed_form(lib, f, u, lam) - ref) <= 20 * EPS * s)


def test_weights_follow_infinite_and_nan_differences(lib):
    """The weights of a stencil with a non-finite difference are numbers (the
    corrections carry the non-finite value to the flux)."""
    bad = np.array([[np.nan, 1.0, 2.0, 3.0], [1.0, np.inf, 2.0, 3.0], [0.0, 0.0, -np.inf, 1e308]])
    w = fixed_weights(lib, list(bad.T))
    assert np.all(np.isfinite(w))


def test_collapsed_weight(lib):
    """W and d(D W)/dD: u and v carry 2^-57 (a reciprocal of 59 bits, a product
    and the truncated indicators), their squares and the sums at most eight times
    that, the last reciprocal 2^-59 and the truncated double 2^-52: 2^-51 in all."""
    rng = np.random.default_rng(5)
    d = np.concatenate([10.0 ** rng.uniform(-12, 12, N), 10.0 ** rng.uniform(-5, -1, N), [0.0, -0.0, 1e300, -1e-300]])
    d *= rng.choice([-1.0, 1.0], d.size)
    w, q = collapsed_weight(lib, d)
    y, a = L(d) * L(d), L(3e-6)
    u, v = a / (a + 4 * y), a / (a + 10 * y)
    den = 1 + 6 * u * u + 3 * v * v
    W = (1 + 2 * u * u - v * v) / den
    A, B = u * u * (1 - u), v * v * (1 - v)
    slope = W - 4 * ((2 * A - B) - W * (6 * A + 3 * B)) / den
    assert np.all(np.abs(L(w) - W) <= 2.0 ** -51 * W)
    assert np.all(np.abs((L(w) - 4 * L(q)) - slope) <= 2.0 ** -49)
