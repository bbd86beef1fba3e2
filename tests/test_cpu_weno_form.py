"""The second-difference form of the WENO5 local Lax-Friedrichs flux that the
order-5 kernels use, in plain float64 against the reference's candidate form
(flux_schemes.H:373-495) in extended precision, on smooth, noisy,
discontinuous and collapsed (first-order fallback) stencils.

Bound: every operation of the kernel's form rounds to within half an ulp of a
quantity bounded by the fluxes' scale s = max |f| + lam max |u|; the chain
from the cell values to the flux has fewer than 40 roundings whose effects
enter with coefficients below 1, so |difference| <= 20 eps s."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps
L = np.longdouble
N = 50000


def reference(f, u, lam):
    f, u, lam = [L(x) for x in f], [L(x) for x in u], L(lam)
    k, e = L(13) / L(12), L(1e-6)

    def edge(a, b, c, d, g):
        b2 = k * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4
        b1 = k * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4
        b0 = k * (c - 2 * d + g) ** 2 + (3 * c - 4 * d + g) ** 2 / 4
        w2, w1, w0 = 1 / (e + b2) ** 2, 6 / (e + b1) ** 2, 3 / (e + b0) ** 2
        num = w2 * (2 * a - 7 * b + 11 * c) + w1 * (-b + 5 * c + 2 * d) + w0 * (2 * c + 5 * d - g)
        return num / (6 * (w2 + w1 + w0))

    return (edge(*f[:5]) + lam * edge(*u[:5])) / 2 + (edge(*f[:0:-1]) - lam * edge(*u[:0:-1])) / 2


def centre(dm, dp):
    t, q = dp - dm, dp + dm
    sc = q * q + ((13.0 / 3.0 * t) * t + 4e-6)
    sa, sb = sc - (8.0 * t) * dm, sc + (8.0 * t) * dp
    return t, sa * sa, sb * sb, sc * sc


def pair(m, c, p):
    x, y, z = c[3] * p[1], m[2] * p[1], m[2] * c[3]
    pp, qq = 2.0 * y + x, 2.0 * y + z
    a, b = x * m[0], z * p[0]
    return (c[0] * pp + (b - 2.0 / 3.0 * a), 3.0 * qq + x), (c[0] * qq + (a - 2.0 / 3.0 * b), 3.0 * pp + z)


def kernel_form(f, u, lam):
    def correction(v, sign):
        c = [centre(v[i + 1] - v[i], v[i + 2] - v[i + 1]) for i in range(4)]
        (nl, dl), (nr, dr) = pair(*c[:3])[0], pair(*c[1:])[1]
        with np.errstate(over="ignore", invalid="ignore"):
            one = (nl * dr + sign * nr * dl) / (dl * dr)
        return np.where(np.maximum(dl, dr) < 2.0 ** 460, one, nl / dl + sign * nr / dr)

    return 0.5 * (f[2] + f[3]) - 0.25 * (correction(f, 1.0) + lam * correction(u, -1.0))


def collapsed_form(f, u, lam):
    d = u[3] - u[2]
    sc = 16.0 / 3.0 * d * d + 4e-6
    sa = 8.0 * d * d + sc
    x, y, z = sc * sc * (sa * sa), 4e-6 ** 2 * (sa * sa), 4e-6 ** 2 * (sc * sc)
    return 0.5 * ((f[2] + f[3]) - lam * d * ((x + 2 * y - z) / (x + 6 * y + 3 * z)))


def stencils(kind, rng):
    if kind == "smooth":
        return 1e5 * (1.0 + 1e-4 * rng.standard_normal((6, N)))
    if kind == "noisy":
        return rng.gamma(2.0, 1.0, (6, N))
    if kind == "shock":
        return np.where(np.arange(6)[:, None] < rng.integers(0, 7, N), 1.0, 0.125) * (1 + 1e-3 * rng.standard_normal((6, N)))
    if kind == "large":
        return 10.0 ** rng.uniform(-3, 17, N) * rng.standard_normal((6, N))
    a, b = rng.standard_normal((2, N)) * 10.0 ** rng.uniform(-6, 6, N)  # collapsed
    return np.stack([a, a, a, b, b, b])


@pytest.mark.parametrize("kind", ["smooth", "noisy", "shock", "large", "collapsed"])
def test_second_difference_form(kind):
    rng = np.random.default_rng(7)
    f, u = stencils(kind, rng), stencils(kind, rng)
    lam = rng.uniform(0.1, 10.0, N)
    ref = reference(f, u, lam)
    s = np.abs(f).max(0) + lam * np.abs(u).max(0)
    assert np.all(np.abs(kernel_form(f, u, lam) - ref) <= 20 * EPS * s)
    if kind == "collapsed":
        assert np.all(np.abs(collapsed_form(f, u, lam) - ref) <= 20 * EPS * s)
