"""The shared-memory layout of a Krylov launch (adhv8_kraken_b200/csrc/sw2_layout.h) compiled as host
C++: the ring depth that fits, the fall-back to none, what a layout keeps as instances come and go,
and that instances solved without the staged sweeps (banded, D-ILU) do not turn them off."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "adhv8_kraken_b200", "csrc")
SHIM = r"""
#include "sw2_layout.h"
using namespace sw2;
extern "C" void layout(int n, const int* needs, int want, int groups, long limit, int* last) {
    std::vector<RingNeed> v;
    for (int i = 0; i < n; i++)
        v.push_back(RingNeed{needs[4 * i] != 0, (unsigned)needs[4 * i + 1], (unsigned)needs[4 * i + 2], needs[4 * i + 3] != 0});
    RingLayout l;
    l.stages = last[0]; l.stage_bytes = last[1]; l.x_bytes = last[2]; l.smem = last[3];
    l = ring_layout(v, want, groups, limit, l);
    last[0] = l.stages; last[1] = l.stage_bytes; last[2] = l.x_bytes; last[3] = (int)l.smem;
}
"""


@pytest.fixture(scope="module")
def layout():
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    work = os.path.join(ROOT, "_build", "layout")
    os.makedirs(work, exist_ok=True)
    src, so = os.path.join(work, "shim.cpp"), os.path.join(work, "liblayout.so")
    with open(src, "w") as fh:
        fh.write(SHIM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", CSRC, "-o", so, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    lib = C.CDLL(so)

    def call(needs, want=-1, last=(0, 0, 0, 0), limit=218 * 1024):
        flat = [x for n in needs for x in n]
        a, b = (C.c_int * max(len(flat), 1))(*flat), (C.c_int * 4)(*last)
        lib.layout(len(needs), a, want, 5, C.c_long(limit), b)
        return tuple(b)
    yield call
    shutil.rmtree(work, ignore_errors=True)


BASIN = (1, 14700, 20096, 1)        # a block-Jacobi instance: record, operand buffer, shares fit
BANDED = (0, 0, 0, 0)               # solved without them


def test_depths(layout):
    stages, stage, x, smem = layout([BASIN])
    assert (stages, stage, x) == (3, 14720, 20096) and smem == 10 * 14720 + 20096
    assert layout([BASIN], want=2) == (2, 14720, 20096, 5 * 14720 + 20096)
    assert layout([BASIN], want=0) == (0, 0, 0, 0)
    assert layout([(1, 30000, 20096, 1)])[0] == 2          # ten records do not fit
    assert layout([(1, 60000, 20096, 1)]) == (0, 0, 0, 0)  # nor do five
    assert layout([BASIN, (1, 14700, 1000, 0)]) == (0, 0, 0, 0)


def test_other_solvers_leave_it_alone(layout):
    assert layout([BASIN, BANDED]) == layout([BASIN]) == layout([BANDED, BASIN])
    assert layout([BANDED])[0] == 3


def test_kept_sizes(layout):
    big = layout([(1, 20000, 40000, 1)])
    assert big[0] == 2
    assert layout([BASIN], last=big)[1:3] == big[1:3]
    # sizes kept from instances that left never turn the sweeps off
    kept = layout([(1, 40000, 1024, 1)])
    assert kept[0] == 2
    assert layout([(1, 14700, 60032, 1)], last=kept) == layout([(1, 14700, 60032, 1)])
