"""Cut cells of boxes that are tiles of one array: each tile's cells are those of
the whole box, bitwise, in one call or tile by tile, with the cache and without."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import Level
from helpers import perturb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cache", [1, 0])
@pytest.mark.parametrize("one_call", [True, False])
def test_tiles_of_one_array(cache, one_call):
    c = perturb(cases.porous_ib(n=24, order=2), 4, vel_amp=1e-2)
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(c.params)))
    abi.check("cache", lib.mfg_set_cutcell_cache(cache))
    g, out = C.byref(c.geom), []
    try:
        for cuts in ([0, 24], [0, 7, 16, 24]):
            lev = Level(c.boxes, c.ncomp, backend="torch", device="cuda")
            lev.set_state(c.state)
            abi.check("fill", lib.mfg_fill_patch(lev.descriptors(), 1, g, 1, 0.0, None))
            n = len(cuts) - 1
            tiles = (abi.Box * n)(*[lev.descriptors()[0] for _ in range(n)])
            for t in range(n):
                tiles[t].lo[2], tiles[t].hi[2] = cuts[t], cuts[t + 1] - 1
            for _ in range(2):  # the entries are built, then applied
                if one_call:
                    abi.check("cut", lib.mfg_cutcells(tiles, n, g, 0.0, None))
                else:
                    for t in range(n):
                        abi.check("cut", lib.mfg_cutcells(C.byref(tiles[t]), 1, g, 0.0, None))
            torch.cuda.synchronize()
            out.append(lev.sborder[0].cpu().numpy())
    finally:
        abi.check("cache", lib.mfg_set_cutcell_cache(1))
    assert np.array_equal(*out)
