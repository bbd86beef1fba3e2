"""Physical-boundary ghost cells filled in one launch: every combination of
wall, extrapolated and user-state boundaries over the three directions, so that
edges and corners go through chains of one to three steps, on several small
boxes, against the oracle's staged fill.  Copies and sign changes are exact; a
user state takes fewer than 64 FP64 operations."""
import ctypes as C
import itertools

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level, chop, geometry
import oracle_lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

KINDS = (abi.BC_WALL, abi.BC_FOEXTRAP, abi.BC_EXT_DIR)


def _case(kinds):
    P = cases.catalyst(n=8, order=5, max_grid=8).params
    ext = (abi.EXT_VELOCITY_INLET, abi.EXT_PRESSURE_OUTLET, abi.EXT_FIXED_STATE)
    for d in range(3):
        P.bc_lo[d], P.bc_hi[d] = kinds[d], KINDS[(KINDS.index(kinds[d]) + 1 + d) % 3]
        for h, e in enumerate((P.ext_lo[d], P.ext_hi[d])):
            e.kind = ext[(d + h) % 3]
            e.dens, e.pres = 0.7 + d, 1e5 * (1 + h)
            for a in range(3):
                e.vel[a] = 0.5 * a - d
            for s in range(P.nspec):
                e.spec[s] = 1.0 + s + h
            for c in range(abi.FLO_NVARS + P.nspec):
                e.state[c] = 0.25 * c + d
            e.keep_interior_pres = h
    return P


@pytest.mark.parametrize("kinds", list(itertools.product(KINDS, repeat=3)))
def test_chain_matches_staged_fill(kinds):
    n, nc = (6, 5, 7), None
    P = _case(kinds)
    nc = abi.FLO_NVARS + P.nspec
    g = geometry((0, 0, 0), tuple(m - 1 for m in n), (0, 0, 0), (1.0, 1.0, 1.0), (0, 0, 0))
    boxes = chop((0, 0, 0), [m - 1 for m in n], 4)
    S = np.random.default_rng(3).uniform(0.5, 2.0, size=(nc,) + n[::-1])
    S[abi.RHOU:abi.RHOW + 1] -= 1.0
    S[abi.VELX:abi.VELZ + 1] -= 1.0
    S[abi.VFRAC] = 1.0
    ref = Level(boxes, nc)
    ref.set_state(S, which="old")
    lib = oracle_lib.load("strict")
    assert lib.oracle_fill_patch(C.byref(P), C.byref(g), ref.descriptors(), len(boxes), 0, 0.0) == 0
    gpu = abi.load()
    abi.check("init", gpu.mfg_init(C.byref(P)))
    lev = Level(boxes, nc, backend="torch", device="cuda")
    lev.set_state(S, which="old")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    abi.check("fill", gpu.mfg_fill_patch(lev.descriptors(), len(boxes), C.byref(g), 0, 0.0, st))
    torch.cuda.synchronize()
    for b in range(len(boxes)):
        want, got = ref.sborder_host(b), lev.sborder_host(b)
        if abi.BC_EXT_DIR not in list(P.bc_lo) + list(P.bc_hi):
            assert np.array_equal(got, want), b
        assert np.all(np.abs(got - want) <= 64 * 2.0 ** -53 * np.abs(want)), b
