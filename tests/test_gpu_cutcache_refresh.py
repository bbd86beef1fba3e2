"""Stored cut-cell weights under every kind of volume-fraction change between
mfg_cutcells calls, for single boxes and lists: values moved by an ulp or by
tens of percent with the same gas, cut and solid cells (weights refreshed in
place), cells that change between the three kinds (entry out of use), and
back.  Each call's Sborder is bitwise that of the same sequence with the cache
off."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level
from helpers import perturb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def edits(rng, vf):
    cut = (vf > 0) & (vf < 1)
    yield vf
    yield vf  # unchanged: stored entries
    yield np.where(cut, np.nextafter(vf, 0.0), vf)
    moved = np.where(cut, np.clip(vf * rng.uniform(0.7, 1.3, vf.shape), 0.01, 0.99), vf)
    yield moved
    yield moved
    other = moved.copy()
    pick = rng.random(vf.shape) < 0.02
    other[pick] = rng.choice([0.0, 0.4, 1.0], size=int(pick.sum()))
    yield other
    yield np.where((other > 0) & (other < 1), np.nextafter(other, 0.0), other)
    yield vf
    yield np.where(cut, np.nextafter(vf, 1.0), vf)


@pytest.mark.parametrize("max_grid", [24, 12, 7])
@pytest.mark.parametrize("name", ["porous", "catalyst"])
def test_every_change_equals_the_uncached_call(name, max_grid):
    c = {"porous": lambda: cases.porous_ib(n=24, order=2, max_grid=max_grid),
         "catalyst": lambda: cases.catalyst(n=24, order=5, max_grid=max_grid)}[name]()
    c = perturb(c, 4, vel_amp=1e-2)
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
    g, out = C.byref(c.geom), []
    for cache in (0, 1):
        abi.check("cache", lib.mfg_set_cutcell_cache(cache))
        lev = Level(c.boxes, c.ncomp, backend="torch", device="cuda")
        d, n = lev.descriptors(), len(c.boxes)
        res = []
        for vf in edits(np.random.default_rng(2), c.state[abi.VFRAC].copy()):
            S = c.state.copy()
            S[abi.VFRAC] = vf
            lev.set_state(S)
            abi.check("fill", lib.mfg_fill_patch(d, n, g, 1, 0.0, None))
            abi.check("cut", lib.mfg_cutcells(d, n, g, 0.0, None))
            torch.cuda.synchronize()
            res.append([x.cpu().numpy() for x in lev.sborder])
        out.append(res)
    abi.check("cache", lib.mfg_set_cutcell_cache(1))
    for k, (a, b) in enumerate(zip(*out)):
        for x, y in zip(a, b):
            assert np.array_equal(x, y), k
