"""Ghost cells of refined boxes from coarse data that exercises every branch of
the interpolation: extrema and sign changes (zero slopes), steep gradients
(slopes cut by the neighbours' bounds) and zeros; and boundary stages of boxes
that touch the domain in none to three directions.  Compared with the oracle's
multi-level step."""
import ctypes as C

import numpy as np
import pytest

from mesoflow_gb300 import abi, cases
from mesoflow_gb300.level import MultiLevel
from oracle_run import OracleAmr

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _step(amr, dt, mode):
    lib = abi.load()
    abi.check("mfg_init", lib.mfg_init(C.byref(amr.params)))
    s = torch.cuda.Stream()
    ml = MultiLevel(amr, backend="torch", device="cuda")
    h = C.c_void_p()
    g = ml.geoms()
    abi.check("create", lib.mfg_boxlist_create(ml.descriptors(), len(amr.boxes), g, len(amr.geoms), C.byref(h)))
    with torch.cuda.stream(s):
        abi.check("step", lib.mfg_boxlist_step_amr(h, 0.0, dt, mode, C.c_void_p(s.cuda_stream)))
    s.synchronize()
    lib.mfg_boxlist_destroy(h)
    return [ml.box_state(b) for b in range(len(amr.boxes))]


def _amr(nlev, seed, noise):
    amr = cases.catalyst_amr(n0=32, nlev=nlev, order=5, blocking=8, max_grid=16, base_grid=16, nspheres=6)
    rng = np.random.default_rng(seed)
    sp = abi.FLO_NVARS
    for s in amr.states:
        gas = s[abi.VFRAC] == 1.0
        for q in range(8):  # gas species: noise and a few exact zeros
            f = 1.0 + noise * rng.standard_normal(gas.shape)
            f[rng.uniform(size=gas.shape) < 0.02] = 0.0
            s[sp + q] *= np.where(gas & (q > 0), np.maximum(f, 0.0), 1.0)
    return amr


@pytest.mark.parametrize("nlev", [2, 3])
def test_noisy_coarse_data_matches_oracle(nlev):
    """One coarse step to the one-step parity tolerance, 1e-12 of each
    component's scale (of the vector's for momenta and velocities)."""
    amr = _amr(nlev, 3 + nlev, 0.2)
    dt = 1e-10
    got = _step(amr, dt, 1)
    o = OracleAmr(amr)
    o.advance(dt)
    want = [o.box_state(b) for b in range(len(amr.boxes))]
    vec = [(abi.RHOU, abi.RHOV, abi.RHOW), (abi.VELX, abi.VELY, abi.VELZ)]
    for c in range(want[0].shape[0]):
        grp = next((v for v in vec if c in v), (c,))
        sc = max(np.abs(w[q]).max() for w in want for q in grp)
        err = max(np.abs(a[c] - w[c]).max() for a, w in zip(got, want))
        assert err <= 1e-12 * sc, (c, err / sc)
