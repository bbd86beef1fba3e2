"""The fixed-point reciprocal, reciprocal square root and limiter half of
mfg_fixed.cuh, compiled for the host, against extended precision, and the
forms of the AUSM+-up splits the face kernels use against the reference's
(flux_schemes.H:107-181).

Bounds: 59 correct bits, rounded once to 53: relative error below 2^-53 (half
an ulp of a significand of 1) plus 2^-58.  The split forms: chains of fewer
than 16 roundings of quantities below 4 (|M| <= 1, |alpha| <= 3/4)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
L = np.longdouble
BOUND = 2.0 ** -53 + 2.0 ** -58

SHIM = r"""
#include "mfg_fixed.cuh"
using namespace mfg;
extern "C" void run(int what, const double* a, const double* b, double* o, int n) {
    for (int i = 0; i < n; ++i)
        o[i] = what == 0 ? rcp_mid(a[i]) : what == 1 ? rsqrt_mid(a[i]) : what == 2 ? limited_half(a[i], b[i])
                                                                        : (double)mid_positive(a[i]);
}
// exp(-(a/den)/b); -1 where the fixed point is not taken
extern "C" void arrhenius(const double* a, double den, const double* b, double* o, int n) {
    for (int i = 0; i < n; ++i)
        if (!mid_positive(a[i]) || !mid_positive(b[i]) || !exp_neg_over(exp_scale(a[i], den), b[i], o + i)) o[i] = -1.0;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src, so = str(d / "f.cpp"), str(d / "f.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mesoflow_gb300", "csrc"), src, "-o", so],
                   check=True, capture_output=True)
    lib = C.CDLL(so)

    def call(what, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = a if b is None else np.ascontiguousarray(b, dtype=np.float64)
        o = np.empty_like(a)
        p = [x.ctypes.data_as(C.c_void_p) for x in (a, b, o)]
        lib.run(C.c_int(what), p[0], p[1], p[2], C.c_int(a.size))
        return o

    call.lib = lib
    return call


def positives(rng, n=200000):
    m = 1.0 + rng.random(n)
    m[::50] = 1.0                          # powers of two and their neighbours
    m[1::50] = np.nextafter(1.0, 2.0)
    m[2::50] = np.nextafter(2.0, 1.0)
    return np.ldexp(m, rng.integers(-980, 975, n))


def test_reciprocal_and_square_root(run):
    x = positives(np.random.default_rng(1))
    assert np.all(run(3, x) == 1.0)
    r = L(1) / L(x)
    assert np.all(np.abs(run(0, x) - r) <= BOUND * r)
    s = L(1) / np.sqrt(L(x))
    assert np.all(np.abs(run(1, x) - s) <= BOUND * s)
    odd = np.array([0.0, -0.0, -1.0, 1e-310, 1e308, np.inf, -np.inf, np.nan, -np.nan])
    assert np.all(run(3, odd) == 0.0)      # these take the FP64 forms


def test_limited_half(run):
    rng = np.random.default_rng(2)
    n = 200000
    a = np.ldexp(1.0 + rng.random(n), rng.integers(-300, 300, n))
    b = np.where(rng.random(n) < 0.5, a * (1.0 + rng.uniform(-0.5, 0.5, n)),
                 a * np.ldexp(1.0 + rng.random(n), rng.integers(-70, 70, n)))
    b[::20] = a[::20]
    b[1::20] = np.nextafter(a[1::20], np.inf)
    h = L(a) * L(b) / (L(a) + L(b))
    got = run(2, a, b)
    assert np.all(np.abs(got - h) <= BOUND * h)
    assert np.array_equal(run(2, b, a), got)                     # symmetric
    assert np.array_equal(run(2, -a, -b), -got)                  # odd
    assert np.all(run(2, a, -b) == 0.0) and np.all(run(2, -a, b) == 0.0)
    z = np.zeros_like(a)
    assert np.all(run(2, a, z) == 0.0) and np.all(run(2, -z, -a) == 0.0) and np.all(run(2, z, z) == 0.0)
    for bad in (np.nan, np.inf, -np.inf):
        assert np.all(np.isnan(run(2, a[:100], np.full(100, bad))))


def test_ausm_split_forms():
    rng = np.random.default_rng(3)
    M = np.concatenate([rng.uniform(-1, 1, 100000), rng.uniform(-3, 3, 100000), [0.0, 1.0, -1.0]])
    alpha = rng.uniform(-0.75, 0.1875, M.size)
    q = M * M - 1.0
    for sign in (1.0, -1.0):
        a = M + sign
        sq, q2 = a * a, q * q
        sub = np.abs(M) <= 1.0
        on = M * sign > 0.0
        m4 = np.where(sub, 0.5 * q2 + sq, np.where(on, 4.0 * sign * M, 0.0))
        g = np.where(sub, sq * (2.0 - sign * M), np.where(on, 4.0, 0.0))
        mq = np.where(sub, M * q2, 0.0)
        # the reference: M4 = sign ((M + sign)^2/4 + (M^2-1)^2/8), P5 = (M + sign)^2 (2 - sign M)/4 + sign alpha M (M^2-1)^2
        m, al = L(M), L(alpha)
        mach = np.where(sub, sign * (0.25 * (m + sign) ** 2 + 0.125 * (m * m - 1) ** 2), 0.5 * (m + sign * np.abs(m)))
        pres = np.where(sub, 0.25 * (m + sign) ** 2 * (2 - sign * m) + sign * al * m * (m * m - 1) ** 2,
                        0.5 * (1 + sign * np.sign(m)))
        tol = 16 * 4 * 2.0 ** -53
        assert np.all(np.abs(sign * 0.25 * m4 - mach) <= tol * np.maximum(1.0, np.abs(M)))
        assert np.all(np.abs((sign * alpha * mq + 0.25 * g) - pres) <= tol)


@pytest.mark.skipif(np.finfo(L).nmant < 63, reason="needs extended precision")
@pytest.mark.parametrize("lo,hi", [(1e-12, 1e-3), (1e-3, 1e2), (1e2, 1e5), (1e5, 3e6)])
def test_arrhenius_factor(run, lo, hi):
    """exp(-x), x = Ea/(RU T): y = x log2(e) has 58.5 bits (the reciprocal's 59
    and two truncations), which the exponential turns into x 2^-58; the series,
    its table and its products leave 2^-57; one rounding."""
    rng = np.random.default_rng(7)
    n, RU = 200000, 8.31446261815324
    Ea = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    T = rng.uniform(150.0, 4000.0, n)
    T[:100] = 2.0 ** rng.integers(6, 12, 100)
    T[100:200] = np.nextafter(T[:100], 0.0)
    o = np.empty(n)
    p = [v.ctypes.data_as(C.c_void_p) for v in (Ea, T, o)]
    run.lib.arrhenius(p[0], C.c_double(RU), p[1], p[2], C.c_int(n))
    x = L(Ea) / L(RU) / L(T)
    taken = o >= 0.0
    assert np.all(taken[x < 354.0]) and not np.any(taken[x > 710.0])
    want = np.exp(-x[taken])
    assert np.all(np.abs(L(o[taken]) - want) <= (2.0 ** -53 + 2.0 ** -57 + x[taken] * 2.0 ** -58) * want)
