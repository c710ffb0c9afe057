"""The search for sub-ranges in the share tables (adhv8_kraken_b200/csrc/sw2_halo.h, compiled as host
C++): it refuses (nsub = 0) only where single tiles do not fit, whatever the number of tiles of a
virtual CTA."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "adhv8_kraken_b200", "csrc")
SHIM = r"""
#include "sw2_halo.h"
extern "C" int nsub(int V, const int* rp, const int* col, int vgrid, int cap, int* max_rows) {
    sw2::HaloTables t;
    sw2::build_halo(V, rp, col, vgrid, cap, t);
    *max_rows = t.max_rows;
    return t.nsub;
}
"""


@pytest.fixture(scope="module")
def lib():
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    work = os.path.join(ROOT, "_build", "halo_search")
    os.makedirs(work, exist_ok=True)
    src, so = os.path.join(work, "shim.cpp"), os.path.join(work, "libhalosearch.so")
    with open(src, "w") as fh:
        fh.write(SHIM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", CSRC, "-o", so, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    yield C.CDLL(so)
    shutil.rmtree(work, ignore_errors=True)


@pytest.mark.parametrize("vgrid", [1, 2, 3])
@pytest.mark.parametrize("tiles", range(1, 33))
def test_single_tiles_that_fit_are_found(lib, tiles, vgrid):
    """A chain (each row refers to the one before and after): a tile and its two halo rows make 34
    rows, two tiles 66, so a cap of 40 needs one tile per sub-range, and a cap of 33 has none."""
    V = 32 * tiles * vgrid
    cols = [[j for j in (i - 1, i + 1) if 0 <= j < V] for i in range(V)]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    col = np.array([j for c in cols for j in c], np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    rows = C.c_int()
    assert lib.nsub(V, p(rp), p(col), vgrid, 40, C.byref(rows)) == tiles and rows.value <= 34
    if tiles > 2:
        assert lib.nsub(V, p(rp), p(col), vgrid, 33, C.byref(rows)) == 0
