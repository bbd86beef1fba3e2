"""Two geometries in turn through one set of arrays, with values that move in
between: every call's Sborder is bitwise that of the same sequence with the
cut-cell cache off, box by box and in one list."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level
from helpers import perturb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def sequence(vf):
    rng = np.random.default_rng(7)
    other = vf.copy()
    pick = rng.random(vf.shape) < 0.02
    other[pick] = rng.choice([0.0, 0.4, 1.0], size=int(pick.sum()))
    for k in range(4):
        for v in (vf, other):
            cut = (v > 0) & (v < 1)
            yield v if k == 0 else np.where(cut, np.clip(v * (1 + 0.05 * k * rng.standard_normal(v.shape)), 0.01, 0.99), v)
    yield vf
    yield vf


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("name", ["porous", "catalyst"])
def test_geometries_in_turn(name, single):
    c = {"porous": lambda: cases.porous_ib(n=24, order=2, max_grid=12),
         "catalyst": lambda: cases.catalyst(n=24, order=5, max_grid=12)}[name]()
    c = perturb(c, 4, vel_amp=1e-2)
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
    g, out = C.byref(c.geom), []
    try:
        for cache in (0, 1):
            abi.check("cache", lib.mfg_set_cutcell_cache(cache))
            lev = Level(c.boxes, c.ncomp, backend="torch", device="cuda")
            d, n = lev.descriptors(), len(c.boxes)
            res = []
            for k, vf in enumerate(sequence(c.state[abi.VFRAC].copy())):
                S = c.state.copy()
                S[abi.VFRAC] = vf
                lev.set_state(S)
                abi.check("fill", lib.mfg_fill_patch(d, n, g, 1, 0.0, None))
                for b in range(n) if single else [None]:
                    abi.check("cut", lib.mfg_cutcells(d if b is None else C.byref(d[b]), n if b is None else 1, g, 0.0, None))
                torch.cuda.synchronize()
                res.append([x.cpu().numpy() for x in lev.sborder])
            out.append(res)
    finally:
        abi.check("cache", lib.mfg_set_cutcell_cache(1))
    for k, (a, b) in enumerate(zip(*out)):
        for x, y in zip(a, b):
            assert np.array_equal(x, y), k
