"""Order-5 fluxes of species whose values differ by many orders of magnitude
across a front: on the low side a face's flux keeps its own digits, whatever the
cells beyond the front hold.  Per face, against the oracle's candidate form, to
1e-12 of the parts that make the flux up (the nonlinear weights times the
candidates' absolute terms, of the Euler flux and of lam times the state), not
of the domain's maximum."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level, geometry
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = abi.NGROW
LOW = [1e-9, 0.0, 1e-13, 1e-4]


def state(P, n, seed):
    """Species 0 everywhere, the others on one side of a front normal to x, y or
    z, or in a layer of three cells, low on the other side."""
    rng = np.random.default_rng(seed)
    shape = tuple(q + 2 * G for q in n[::-1])
    idx = dict(zip("zyx", np.indices(shape)))
    noise = lambda a: 1.0 + a * rng.standard_normal(shape)
    spec = [30.0 * noise(0.01)]
    for s, ax in enumerate("xyzx", 1):
        at = G + n["xyz".index(ax)] // 2
        high = (idx[ax] >= at) & ((idx[ax] < at + 3) | (s != 4))
        spec.append(np.where(high, 8.0 * s, LOW[s - 1]) * noise(0.01))
    rho = sum(spec[s] * P.molwt[s] for s in range(P.nspec))
    vel = [20.0 * (0.4 + 0.3 * rng.standard_normal(shape)) for _ in range(3)]
    return cases.state_from_prim(P, rho, *vel, 1e5 * noise(0.01), spec, np.ones(shape))


def parts(v):
    """Sum of the two edges' weighted absolute candidates over the faces of the
    last axis (cells padded by three)."""
    m = v.shape[-1] - 5
    c = [v[..., q:q + m] for q in range(6)]

    def edge(a, b, c, d, e):
        w = [1.0 / (1e-6 + 13 / 12 * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4) ** 2,
             6.0 / (1e-6 + 13 / 12 * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4) ** 2,
             3.0 / (1e-6 + 13 / 12 * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4) ** 2]
        a, b, c, d, e = map(np.abs, (a, b, c, d, e))
        return (w[0] * (2 * a + 7 * b + 11 * c) + w[1] * (b + 5 * c + 2 * d) + w[2] * (2 * c + 5 * d + e)) / (6 * sum(w))

    return edge(*c[:5]) + edge(*c[:0:-1])


def fluxes(P, n, S, backend, boxes):
    geom = geometry((0, 0, 0), [q - 1 for q in n], (0, 0, 0), [0.01 * q for q in n], (0, 0, 0))
    lev = Level(boxes, S.shape[0], backend=backend, device="cuda", with_flux=True)
    for b, (lo, hi) in enumerate(boxes):
        lev.set_sborder(b, S[(slice(None),) + tuple(slice(lo[q], hi[q] + 1 + 2 * G) for q in (2, 1, 0))])
    if backend == "numpy":
        assert oracle_lib.load("strict").oracle_compute_dsdt(C.byref(P), C.byref(geom), lev.descriptors(), len(boxes)) == 0
        return lev.flux
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(P)))
    abi.check("dsdt", lib.mfg_compute_dsdt_flow(lev.descriptors(), len(boxes), C.byref(geom), 0.0, 1e-6, None))
    torch.cuda.synchronize()
    return [[f.cpu().numpy() for f in b] for b in lev.flux]


def params():
    P = cases.taylor_green_mix(n=8).params
    for s in range(P.nspec):
        P.diff_gas[s] = 0.0  # the hyperbolic flux alone
    return P


# the per-face form, then the column sweep (more threads than fill the GPU)
@pytest.mark.parametrize("n", [(9, 8, 7), (40, 36, 33)])
def test_low_side_of_a_front(n):
    P = params()
    S = state(P, n, sum(n))
    whole = [((0, 0, 0), tuple(q - 1 for q in n))]
    want, got = (fluxes(P, n, S, k, whole)[0] for k in ("numpy", "torch"))
    lam = 2.0 * np.sqrt(1.67 * S[abi.PRES].max() / S[abi.RHO].min())
    for d in range(3):
        for s in range(1, P.nspec):
            ax = 2 - d
            cut = tuple(slice(None) if a == ax else slice(G, -G) for a in range(3))
            u, v = (np.moveaxis(S[c][cut], ax, -1) for c in (abi.FLO_NVARS + s, abi.VELX + d))
            scale = np.moveaxis(parts(u * v) + lam * parts(u), -1, ax)
            e = np.abs(got[d][abi.FLO_NVARS + s] - want[d][abi.FLO_NVARS + s])
            assert np.all(e <= 1e-12 * scale), (d, s)  # both zero where the whole stencil is


def test_forms_agree_beside_fronts():
    """The column sweep of one box and the per-face form of its parts, bitwise."""
    n = (40, 36, 33)
    P = params()
    S = state(P, n, 5)
    whole = fluxes(P, n, S, "torch", [((0, 0, 0), tuple(q - 1 for q in n))])[0]
    lo = (G + 8, G + 7, G + 5)
    part = [((lo[0], lo[1], lo[2]), (lo[0] + 17, lo[1] + 16, lo[2] + 15))]
    box = fluxes(P, n, S, "torch", part)[0]
    for d in range(3):
        sub = whole[d][(slice(None),) + tuple(slice(part[0][0][q], part[0][1][q] + 1 + (q == d)) for q in (2, 1, 0))]
        assert np.array_equal(box[d], sub), d


def test_batched_step_beside_fronts():
    """The batched sweep against the per-box step, bitwise."""
    n = 24
    c = cases.taylor_green_mix(n=n, order=5, max_grid=12)
    c.state = state(params(), (n, n, n), 3)[:, G:-G, G:-G, G:-G].copy()
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
    a, b = (Level(c.boxes, c.ncomp, backend="torch", device="cuda") for _ in range(2))
    a.set_state(c.state)
    b.set_state(c.state)
    s = torch.cuda.Stream()
    st = C.c_void_p(s.cuda_stream)
    h = C.c_void_p()
    abi.check("create", lib.mfg_boxlist_create(b.descriptors(), len(c.boxes), (abi.Geom * 1)(c.geom), 1, C.byref(h)))
    with torch.cuda.stream(s):
        abi.check("level", lib.mfg_advance_level(a.descriptors(), len(c.boxes), C.byref(c.geom), 0.0, 1e-6, 0, 1, None, st))
        abi.check("boxlist", lib.mfg_boxlist_step(h, 0.0, 1e-6, 1, st))
    s.synchronize()
    lib.mfg_boxlist_destroy(h)
    assert np.array_equal(a.get_state(c.shape_zyx), b.get_state(c.shape_zyx))
