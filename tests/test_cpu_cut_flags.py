"""The life of a stored cut-cell entry (mfg_cut_flags.h, compiled here for the
host) over random sequences of volume fractions: values that move within their
kind, other geometries, and the stored one coming back.  The entry is applied in
every pass whose gas, cut and solid cells are those it was built for, always with
weights of the pass's own values, and is marked for dropping only after a pass
that could not use it."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N = 12

SHIM = r"""
#include "mfg_cut_flags.h"
using namespace mfg;
// One pass: v the volume fractions, copy the entry's, w the values its weights were computed from.
extern "C" int cut_pass(const double* v, double* copy, double* w, unsigned* flag, int n) {
    for (int i = 0; i < n; ++i) *flag |= vf_change(v[i], copy + i);
    const int apply = vf_apply(*flag);
    if (vf_refresh(*flag))
        for (int i = 0; i < n; ++i) w[i] = v[i];
    *flag = vf_after(*flag);
    return apply;
}
extern "C" int left(unsigned flag) { return (flag & (VF_OTHER | VF_LEFT)) != 0; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("flags")
    src, so = str(d / "f.cpp"), str(d / "f.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mesoflow_gb300", "csrc"), src, "-o", so],
                   check=True, capture_output=True)
    return C.CDLL(so)


def kinds(v):
    return np.where(v == 1.0, 2, np.where((v > 0) & (v < 1), 1, 0))


@pytest.mark.parametrize("seed", range(20))
def test_entry_follows_its_geometry(lib, seed):
    rng = np.random.default_rng(seed)
    geometries = [rng.choice([0.0, 0.3, 0.7, 1.0, 1.0], N) for _ in range(3)]
    built = geometries[0].copy()
    copy, w, flag = built.copy(), built.copy(), C.c_uint(0)
    seen = set()
    for _ in range(200):
        v = geometries[rng.integers(3)].copy()
        cut = (v > 0) & (v < 1)
        move = rng.integers(3)
        if move == 1:
            v = np.where(cut, np.nextafter(v, rng.choice([0.0, 1.0])), v)
        elif move == 2:
            v = np.where(cut & (rng.random(N) < 0.5), v * rng.uniform(0.9, 1.1), v)
        applied = lib.cut_pass(*[x.ctypes.data_as(C.c_void_p) for x in (v, copy, w)], C.byref(flag), C.c_int(N))
        same = bool(np.all(kinds(v) == kinds(built)))
        assert bool(applied) == same
        assert bool(lib.left(flag)) == (not same)
        if applied:
            assert np.array_equal(w.view(np.uint64), v.view(np.uint64))
        seen.add(same)
    assert seen == {True, False}
