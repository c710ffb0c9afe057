"""The closed-form Jacobian of a fully wet element (adhv8_kraken_b200/csrc/sw2_wet_jac.cuh) compiled as
host C++ and compared with the residual it differentiates (sw2_elem_resid, itself bit-identical to
the oracle): Ridders-extrapolated central differences of every column, on random wet elements over
velocities from rest up, depths on and around both floors, with and without drag (clipped and not),
Coriolis, a water source, wind, isotropic viscosity, temporal weights, and Dirichlet rows."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "adhv8_kraken_b200", "csrc")
SHIM = r"""
#include <algorithm>
#include <cmath>
using std::fabs; using std::fmax; using std::log; using std::pow; using std::sqrt;
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#include "sw2_wet_jac.cuh"
using namespace sw2;
static void unpack(const double* g, ElemIn& in) {
    for (int i = 0; i < 3; i++) {
        in.x[i] = g[i]; in.y[i] = g[3 + i]; in.z[i] = g[6 + i]; in.h[i] = g[9 + i]; in.u[i] = g[12 + i]; in.v[i] = g[15 + i];
        in.ho[i] = g[18 + i]; in.uo[i] = g[21 + i]; in.vo[i] = g[24 + i];
        in.hoo[i] = in.ho[i]; in.uoo[i] = in.uo[i]; in.voo[i] = in.vo[i];
    }
    const double cr = (in.x[1] - in.x[0]) * (in.y[2] - in.y[0]) - (in.x[2] - in.x[0]) * (in.y[1] - in.y[0]);
    in.djac = 0.5 * cr;
    for (int i = 0; i < 3; i++) {
        const int j = (i + 1) % 3, k = (i + 2) % 3;
        in.gx[i] = (in.y[j] - in.y[k]) / cr;
        in.gy[i] = (in.x[k] - in.x[j]) / cr;
    }
    in.wsx = g[27]; in.wsy = g[28];
}
static MatParams mat(const double* m) {
    MatParams M{};
    M.ks = m[0]; M.ev_st = 0.0; M.ev_tr = m[1]; M.cor_speed = m[2]; M.water_src = m[3]; M.has_source = m[3] != 0.0;
    return M;
}
extern "C" void resid(const double* g, const double* ph, const double* m, const int* df, double* out) {
    ElemIn in;
    unpack(g, in);
    const PhysParams P{ph[0], ph[1], ph[2], ph[3], ph[4], ph[5]};
    double er[3][3];
    sw2_elem_resid(in, in.h, in.u, in.v, 0, kPertNone, P, mat(m), df, er);
    for (int i = 0; i < 3; i++) { out[3 * i] = er[i][1]; out[3 * i + 1] = er[i][2]; out[3 * i + 2] = er[i][0]; }
}
extern "C" void jac(const double* g, const double* ph, const double* m, const int* df, double* out) {
    ElemIn in;
    unpack(g, in);
    WetElem E;
    for (int i = 0; i < 3; i++) {
        E.x[i] = in.x[i]; E.y[i] = in.y[i]; E.z[i] = in.z[i]; E.h[i] = in.h[i]; E.u[i] = in.u[i]; E.v[i] = in.v[i];
        E.ho[i] = in.ho[i]; E.uo[i] = in.uo[i]; E.vo[i] = in.vo[i]; E.gx[i] = in.gx[i]; E.gy[i] = in.gy[i];
    }
    E.djac = in.djac; E.wsx = in.wsx; E.wsy = in.wsy;
    const PhysParams P{ph[0], ph[1], ph[2], ph[3], ph[4], ph[5]};
    wet_jacobian(E, P, mat(m), df, out);
}
"""


@pytest.fixture(scope="module")
def lib():
    if shutil.which("g++") is None or not os.path.isdir("/usr/local/cuda/include"):
        pytest.skip("no host C++ compiler or CUDA headers")
    work = os.path.join(ROOT, "_build", "wet_jac")
    os.makedirs(work, exist_ok=True)
    src, so = os.path.join(work, "shim.cpp"), os.path.join(work, "libwetjac.so")
    with open(src, "w") as fh:
        fh.write(SHIM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", CSRC, "-I", "/usr/local/cuda/include",
                        "-o", so, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    yield C.CDLL(so)
    shutil.rmtree(work, ignore_errors=True)


def _call(f, g, ph, m, df, n):
    out = np.zeros(n)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    f(p(g), p(ph), p(m), p(df), p(out))
    return out


def _column(lib, g, ph, m, df, k, h0):
    """Central differences of steps h0, h0/2, ..., extrapolated to 0 (Ridders)."""
    def diff(h):
        a, b = g.copy(), g.copy()
        a[k] += h
        b[k] -= h
        return (_call(lib.resid, a, ph, m, df, 9) - _call(lib.resid, b, ph, m, df, 9)) / (a[k] - b[k])
    t = [[diff(h0)]]
    for i in range(1, 4):
        t.append([diff(h0 / 2 ** i)])
        for j in range(1, i + 1):
            t[i].append(t[i][j - 1] + (t[i][j - 1] - t[i - 1][j - 1]) / (4.0 ** j - 1.0))
    return t[-1][-1]


@pytest.mark.parametrize("drag,visc,cor,src,wind,alpha", [
    (0.0, 0.0, 0.0, 0.0, 0.0, 0.0), (0.01, 0.0, 0.0, 0.0, 0.0, 0.0), (90.0, 0.0, 0.0, 0.0, 0.0, 0.0),
    (0.05, 3.0, 1e-4, 0.0, 0.0, 0.5), (0.05, 0.5, -1e-4, 2e-4, 0.3, 0.0)])
def test_closed_form_equals_extrapolated_differences(lib, drag, visc, cor, src, wind, alpha):
    rng = np.random.default_rng(17)
    ph = np.array([9.81, 0.1, 0.4, alpha, 0.5, 5.0])
    m = np.array([drag, visc, cor, src])
    df = np.zeros(3, np.int32)
    for trial in range(60):
        g = np.zeros(29)
        ang = np.sort(rng.uniform(0, 2 * np.pi, 3))
        if np.min(np.diff(np.append(ang, ang[0] + 2 * np.pi))) < 0.5:
            continue
        g[0:3], g[3:6] = 20 * np.cos(ang), 20 * np.sin(ang)
        g[6:9] = rng.uniform(-1, 1, 3)
        deep = trial % 3 != 0   # the others stay below both floors
        g[9:12] = rng.uniform(0.8, 6.0, 3) if deep else rng.uniform(0.02, 0.08, 3)
        g[12:18] = rng.uniform(0.05, 1.5, 6) * rng.choice([-1, 1], 6)
        g[18:21] = g[9:12] * rng.uniform(0.95, 1.05, 3)
        g[21:27] = g[12:18] + rng.uniform(-0.05, 0.05, 6)
        g[27:29] = wind
        J = _call(lib.jac, g, ph, m, df, 81).reshape(3, 3, 3, 3)      # a, b, row, var
        scale = np.abs(J).max()
        for b in range(3):
            for var, off in enumerate((12, 15, 9)):
                k = off + b
                col = _column(lib, g, ph, m, df, k, 0.02 * abs(g[k])).reshape(3, 3)   # a, row
                # steps of 2 % and 2.5e-3 of the value: the extrapolated remainder and the
                # residual's rounding over the step are both below 1e-9 of the largest entry
                assert np.abs(J[:, b, :, var] - col).max() <= 1e-8 * scale, (trial, b, var)


def test_at_rest_on_the_floors_and_dirichlet_rows(lib):
    """The reference's own difference quotients: at rest, with depths exactly on the floors, and with
    held rows."""
    ph = np.array([9.81, 0.1, 0.4, 0.0, 0.5, 5.0])
    m = np.array([0.02, 1.0, 0.0, 0.0])
    p = 1.4901161193847656e-08
    for depth in (0.1, 0.4, 2.0):
        for df in (np.zeros(3, np.int32), np.array([1, 2, 4], np.int32)):
            g = np.zeros(29)
            g[0:3], g[3:6] = (0.0, 30.0, 5.0), (0.0, 2.0, 25.0)
            g[6:9] = (0.0, 0.1, -0.2)
            g[9:12] = g[18:21] = depth
            J = _call(lib.jac, g, ph, m, df, 81).reshape(3, 3, 3, 3)
            scale = np.abs(J).max()
            for b in range(3):
                for var, off in enumerate((12, 15, 9)):
                    k = off + b
                    eps = max(abs(g[k]) * (1 + p) - abs(g[k]), p)
                    a, c = g.copy(), g.copy()
                    a[k] += eps
                    c[k] -= eps
                    q = (_call(lib.resid, a, ph, m, df, 9) - _call(lib.resid, c, ph, m, df, 9)) / (2 * eps)
                    # the quotient's own rounding: the residual's terms over the step
                    assert np.abs(J[:, b, :, var] - q.reshape(3, 3)).max() <= 1e-6 * scale, (depth, b, var)
