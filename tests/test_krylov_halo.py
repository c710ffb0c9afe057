"""The share tables of the Krylov solve (adhv8_kraken_b200/csrc/sw2_halo.h) compiled as host C++:
every row in exactly one sub-range, every block's column found again through its buffer number, the
halo rows external, ascending and without repeats, and no buffer above the cap -- on banded, random
and fan patterns, with row counts around the tile size, with virtual grids from one to one per tile,
and the refusal (nsub = 0) where a single tile needs more than the cap."""
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
extern "C" int halo_build(int V, const int* rp, const int* col, int vgrid, int cap, int* max_rows, int* nidx) {
    build_halo(V, rp, col, vgrid, cap, t);
    *max_rows = t.max_rows;
    *nidx = (int)t.idx.size();
    return t.nsub;
}
extern "C" void halo_get(int* ptr, int* idx, unsigned short* lcol) {
    std::copy(t.ptr.begin(), t.ptr.end(), ptr);
    std::copy(t.idx.begin(), t.idx.end(), idx);
    std::copy(t.lcol.begin(), t.lcol.end(), lcol);
}
"""


@pytest.fixture(scope="module")
def halo():
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    work = os.path.join(ROOT, "_build", "halo")
    os.makedirs(work, exist_ok=True)
    src, lib = os.path.join(work, "shim.cpp"), os.path.join(work, "libhalo.so")
    with open(src, "w") as fh:
        fh.write(SHIM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", CSRC, "-o", lib, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    yield C.CDLL(lib)
    shutil.rmtree(work, ignore_errors=True)


def _pattern(kind, V, rng):
    rows = [set() for _ in range(V)]
    for i in range(V):
        if kind == "band":
            js = [i - 1, i + 1, i - 7, i + 7, i + 8]
        elif kind == "random":
            js = rng.integers(0, V, 6)
        else:   # fan: every row refers to row 0, row 0 to every row
            js = [0, i - 1, i + 1]
        for j in js:
            if 0 <= j < V and j != i:
                rows[i].add(int(j))
                rows[int(j)].add(i)
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    return rp, np.array([j for r in rows for j in sorted(r)], np.int32)


@pytest.mark.parametrize("kind,V,vgrid,cap", [
    ("band", 1, 1, 64), ("band", 31, 1, 64), ("band", 32, 1, 64), ("band", 33, 2, 64), ("band", 3001, 94, 96),
    ("band", 3001, 5, 200), ("band", 20000, 444, 1472), ("random", 2000, 63, 1472), ("random", 2000, 7, 400),
    ("random", 2000, 63, 100), ("fan", 1500, 47, 1600), ("fan", 1500, 11, 300)])
def test_share_tables(halo, kind, V, vgrid, cap):
    rp, col = _pattern(kind, V, np.random.default_rng(5))
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    mr, ni = C.c_int(), C.c_int()
    nsub = halo.halo_build(V, p(rp), p(col), vgrid, cap, C.byref(mr), C.byref(ni))
    nt = (V + 31) // 32
    if nsub == 0:   # refused: some tile and what it refers to must exceed the cap
        worst = max(len(set(col[rp[a]:rp[min(a + 32, V)]].tolist()) | set(range(a, min(a + 32, V)))) for a in range(0, V, 32))
        assert worst > cap
        return
    ptr, idx, lcol = np.zeros(vgrid * nsub + 1, np.int32), np.zeros(max(ni.value, 1), np.int32), np.zeros(max(len(col), 1), np.uint16)
    halo.halo_get(p(ptr), p(idx), p(lcol))
    assert mr.value <= cap and ptr[-1] == ni.value
    nxt = 0
    for v in range(vgrid):
        a, b = v * nt // vgrid, (v + 1) * nt // vgrid
        for s in range(nsub):   # as the kernel cuts a virtual CTA's tiles
            r0 = min(V, (a + s * (b - a) // nsub) * 32)
            r1 = min(V, (a + (s + 1) * (b - a) // nsub) * 32)
            assert r0 == nxt
            nxt = r1
            h = idx[ptr[v * nsub + s]:ptr[v * nsub + s + 1]]
            assert np.all(np.diff(h) > 0) and not np.any((h >= r0) & (h < r1))
            assert (r1 - r0) + len(h) <= mr.value
            buf = np.concatenate([np.arange(r0, r1), h])
            assert np.array_equal(buf[lcol[rp[r0]:rp[r1]]], col[rp[r0]:rp[r1]])
    assert nxt == V
