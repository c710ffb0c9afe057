"""The row order of the Krylov solve (build_shares of adhv8_kraken_b200/csrc/sw2_halo.h, compiled as
host C++): a mesh numbered with locality keeps its order and its tables, one without gets the Morton
order of its nodes, with the same blocks in it and tables that hold; coordinates that order nothing
change nothing."""
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
using namespace sw2;
static HaloTables t;
static std::vector<int> rp, col, order;
extern "C" int shares(int V, const int* rp_, const int* col_, const double* x, const double* y, int vgrid, int cap, int* out) {
    rp.assign(rp_, rp_ + V + 1);
    col.assign(col_, col_ + rp_[V]);
    build_shares(V, rp, col, x, y, vgrid, cap, t, order);
    out[0] = t.nsub; out[1] = t.max_rows; out[2] = (int)t.idx.size(); out[3] = (int)order.size();
    return 0;
}
extern "C" int plain_halo(int V, const int* rp_, const int* col_, int vgrid, int cap) {
    HaloTables p;
    build_halo(V, rp_, col_, vgrid, cap, p);
    return (int)p.idx.size();
}
extern "C" void get(int* rp_, int* col_, int* order_, int* ptr, int* idx, unsigned short* lcol) {
    std::copy(rp.begin(), rp.end(), rp_);
    std::copy(col.begin(), col.end(), col_);
    std::copy(order.begin(), order.end(), order_);
    std::copy(t.ptr.begin(), t.ptr.end(), ptr);
    std::copy(t.idx.begin(), t.idx.end(), idx);
    std::copy(t.lcol.begin(), t.lcol.end(), lcol);
}
"""


@pytest.fixture(scope="module")
def lib():
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    work = os.path.join(ROOT, "_build", "order")
    os.makedirs(work, exist_ok=True)
    src, so = os.path.join(work, "shim.cpp"), os.path.join(work, "liborder.so")
    with open(src, "w") as fh:
        fh.write(SHIM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", CSRC, "-o", so, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    yield C.CDLL(so)
    shutil.rmtree(work, ignore_errors=True)


def _grid(nx, ny, perm):
    """Off-diagonal pattern and coordinates of a triangulated grid, node perm[k] at number k."""
    at = np.empty(nx * ny, int)
    at[perm] = np.arange(nx * ny)
    i, j = np.divmod(perm, ny)
    cols = []
    for a, b in zip(i, j):
        near = [(a - 1, b), (a + 1, b), (a, b - 1), (a, b + 1), (a - 1, b - 1), (a + 1, b + 1)]
        cols.append(sorted(at[p * ny + q] for p, q in near if 0 <= p < nx and 0 <= q < ny))
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    return rp, np.concatenate(cols).astype(np.int32), i.astype(float), j.astype(float)


def _call(lib, rp, col, x, y, vgrid, cap):
    V = len(rp) - 1
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    out = np.zeros(4, np.int32)
    lib.shares(V, p(rp), p(col), p(x), p(y), vgrid, cap, p(out))
    nsub, max_rows, nidx, nord = (int(v) for v in out)
    a = [np.zeros(V + 1, np.int32), np.zeros(len(col), np.int32), np.zeros(max(nord, 1), np.int32),
         np.zeros(vgrid * max(nsub, 1) + 1, np.int32), np.zeros(max(nidx, 1), np.int32), np.zeros(len(col), np.uint16)]
    lib.get(*(p(v) for v in a))
    return nsub, max_rows, a[0], a[1], a[2][:nord], a[3], a[4][:nidx], a[5], lib.plain_halo(V, p(rp), p(col), vgrid, cap)


@pytest.mark.parametrize("nx,ny,vgrid", [(33, 31, 7), (64, 65, 13), (101, 90, 20)])
def test_a_scattered_numbering_is_reordered(lib, nx, ny, vgrid):
    V = nx * ny
    rp, col, x, y = _grid(nx, ny, np.random.default_rng(nx).permutation(V))
    nsub, max_rows, krp, kcol, order, ptr, idx, lcol, before = _call(lib, rp, col, x, y, vgrid, 1024)
    assert nsub >= 1 and max_rows <= 1024
    assert np.array_equal(np.sort(order), np.arange(V))
    assert 2 * len(idx) <= before
    # every row has the blocks it had, in the order it had them
    for r in range(V):
        old = order[r]
        assert np.array_equal(order[kcol[krp[r]:krp[r + 1]]], col[rp[old]:rp[old + 1]])
    # and each is found again through its buffer number
    nt = (V + 31) // 32
    for v in range(vgrid):
        a, b = v * nt // vgrid, (v + 1) * nt // vgrid
        for s in range(nsub):
            r0, r1 = (min(V, 32 * (a + q * (b - a) // nsub)) for q in (s, s + 1))
            halo = idx[ptr[v * nsub + s]:ptr[v * nsub + s + 1]]
            rows = np.concatenate([np.arange(r0, r1), halo])
            assert np.array_equal(rows[lcol[krp[r0]:krp[r1]]], kcol[krp[r0]:krp[r1]])


@pytest.mark.parametrize("nx,ny,vgrid", [(300, 12, 22), (64, 64, 4), (9, 9, 1), (55, 47, 41)])
def test_a_numbering_with_locality_is_kept(lib, nx, ny, vgrid):
    """The last one has more halo than own rows, but few of either."""
    rp, col, x, y = _grid(nx, ny, np.arange(nx * ny))
    nsub, _, krp, kcol, order, _, idx, _, before = _call(lib, rp, col, x, y, vgrid, 1024)
    assert nsub >= 1 and len(order) == 0 and len(idx) == before
    assert np.array_equal(krp, rp) and np.array_equal(kcol, col)


def test_coordinates_that_order_nothing(lib):
    rp, col, x, y = _grid(40, 40, np.random.default_rng(1).permutation(1600))
    nsub, _, krp, kcol, order, _, idx, _, before = _call(lib, rp, col, 0 * x + 3.0, 0 * y - 1.0, 10, 1024)
    assert nsub >= 1 and len(order) == 0 and len(idx) == before and np.array_equal(kcol, col)
