// sw2_wet_jac.cuh -- the exact Jacobian of a fully wet element's residual.
//
// The reference differences the residual (fe_sw2_load, src/fe/sw2/fe_sw2_load.c:85-142): eighteen
// evaluations per element, each carrying a quotient's and a root's latency chain, for derivatives
// good to about 1e-8.  The residual of a fully wet element (elem_resid_impl<true>) is smooth but for
// two kinks, so its nine columns have closed forms that share almost everything: the averages,
// gradients, drag law and SUPG scales once per element, a dozen products per entry after that.
// The kinks -- the depth floors max(h, dll) and max(h, dul) -- are differenced with the reference's
// step, so a depth that sits exactly on one gives the reference's mean of the two sides.
// The floors under the mean depth in the residual's quotients (FLT_EPSILON and the drag law's 1e-8) are
// left out: an element is on this path only while every depth is above kWetMargin (sw2_kernels.cuh),
// which is higher; thinner films take the general path and its differences.
//
// Used by the Newton iterations of instances whose materials have an isotropic user eddy viscosity
// (the estimated viscosities have a root of the velocity gradients, which is not smooth at rest);
// sw2gpu_load, the unit for parity with fe_sw2_load, keeps the differences.
#pragma once
#include "sw2_physics.cuh"

namespace sw2 {

// what the closed forms need of an element
struct WetElem {
    double x[3], y[3], z[3];
    double h[3], u[3], v[3], ho[3], uo[3], vo[3];
    double djac, gx[3], gy[3];
    double wsx, wsy;
};

// materials the closed forms cover
__host__ __device__ inline bool wet_jac_material(const MatParams& M) { return M.eev_mode == 0 && M.ev_st == 0.0; }

// d/dh of max(h, floor) as the central difference with the reference's step
__device__ __forceinline__ double floor_slope(double h, double floor, double eps) {
    return (fmax(h + eps, floor) - fmax(h - eps, floor)) / (2.0 * eps);
}

// o[(3 a + b) * 9 + 3 row + var]: block (a, b), rows (x-momentum, y-momentum, continuity), columns
// (u, v, h), before the Dirichlet columns are taken out.  dflag: as elem_resid_impl.
__device__ __forceinline__ void wet_jacobian(const WetElem& E, const PhysParams& P, const MatParams& M, const int* dflag,
                                             double* o) {
    const double A = E.djac, dt = P.dt, g = P.g;
    const double Su = E.u[0] + E.u[1] + E.u[2], Sv = E.v[0] + E.v[1] + E.v[2], Sh = E.h[0] + E.h[1] + E.h[2];
    const double ua = Su * kOne3, va = Sv * kOne3, ha = Sh * kOne3;
    const double gux = dot3(E.u, E.gx), guy = dot3(E.u, E.gy), gvx = dot3(E.v, E.gx), gvy = dot3(E.v, E.gy);
    const double ghx = dot3(E.h, E.gx), ghy = dot3(E.h, E.gy), gzx = dot3(E.z, E.gx), gzy = dot3(E.z, E.gy);
    // sum_bc T_abc x_b y_c of the integrals of three linear functions (T = 6, 2, 1 by coincidences)
    auto tri = [](const double* x, const double* y, double X, double Y, double Pxy, int a) {
        return X * Y + Pxy + x[a] * Y + X * y[a] + 2.0 * x[a] * y[a];
    };
    const double Puu = dot3(E.u, E.u), Puv = dot3(E.u, E.v), Pvv = dot3(E.v, E.v), Puh = dot3(E.u, E.h), Pvh = dot3(E.v, E.h);

    // drag law and its slope in the depth (drag_coef)
    double res = 0.0, dres = 0.0;
    if (M.ks > kSmall) {
        const double ks = fmax(M.ks, 1.E-8);
        const bool clipped = ks > 29.7 * ha;
        const double b = clipped ? 1.0 : 29.7 * (ha / ks);
        const double L = log(b + 1.0), den = (b + 1.0) * (L - 1.0) + 1.0, t = .4 * b / den;
        res = 2. * (t * t) / (2.0 * g);
        if (!clipped) dres = 4. * t * (.4 * (den - b * L) / (den * den)) * (29.7 / ks) / (2.0 * g);
    }
    const double wmag = sqrt(ua * ua + va * va), iw = wmag > 0.0 ? 1.0 / wmag : 0.0;
    // SUPG: scales, strong equations
    const double ih = 1.0 / ha, adt = A * dt;
    const double sr2 = ua * ua + va * va + g * ha + kSmall;
    const double tau = P.tau_pg * sqrt(A) / sqrt(sr2), ts = -tau / sr2;
    const double bx = res * ua * wmag, by = res * va * wmag, gih = adt * g * ih;
    const double cs = M.cor_speed, src = M.has_source ? M.water_src : 0.0;
    const double ceq = A * (ha - avg3(E.ho)) + adt * (ua * ghx + ha * gux + va * ghy + ha * gvy) + src * adt;
    const double xeq = A * (ua - avg3(E.uo)) + adt * (ua * gux + va * guy) + adt * g * (ghx + gzx) + gih * bx -
                       adt * (va * cs + E.wsx * ih);
    const double yeq = A * (va - avg3(E.vo)) + adt * (ua * gvx + va * gvy) + adt * g * (ghy + gzy) + gih * by +
                       adt * (ua * cs - E.wsy * ih);
    const double th = tau * ha;
    // friction fluxes per vertex: slopes of u |u| and v |u|
    double fuu[3], fuv[3], fvv[3], fx[3], fy[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double m = sqrt(E.u[i] * E.u[i] + E.v[i] * E.v[i]), im = m > 0.0 ? 1.0 / m : 0.0;
        fx[i] = E.u[i] * m;
        fy[i] = E.v[i] * m;
        fuu[i] = m + E.u[i] * E.u[i] * im;
        fuv[i] = E.u[i] * E.v[i] * im;
        fvv[i] = m + E.v[i] * E.v[i] * im;
    }
    const double sfx = fx[0] + fx[1] + fx[2], sfy = fy[0] + fy[1] + fy[2];
    const double k12 = -adt * kOne12, k60 = -adt * kOne60;
    const double tf = 1. + P.alpha / 2., tc = A * tf * kOne12, tm = A * tf * kOne3;
    const double kf = adt * g * kOne12, kfr = kf * res;
    const double hd = (ha < P.dul) ? P.dul : ha, kd = dt * A * hd * M.ev_tr;
    const double dxx = 2. * M.ev_tr * gux, dxy = M.ev_tr * (guy + gvx), dyy = 2. * M.ev_tr * gvy;
    const double kc = adt * cs * kOne60;
    const double kpf = -0.5 * g * dt * kOne6 * A, kb = A * kOne12 * g * dt, kq = kOne12 * 0.5 * dt * g;
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const double gxb = E.gx[b], gyb = E.gy[b];
        const double tuh = k60 * tri(E.u, E.h, Su, Sh, Puh, b), tvh = k60 * tri(E.v, E.h, Sv, Sh, Pvh, b);
        const double adv = adt * (ua * gxb + va * gyb);
        const double eps = fd_eps(E.h[b]);
        const double mb = fmax(E.h[b], P.dll), ms = floor_slope(E.h[b], P.dll, eps);
        // slopes of tau, the scales and the strong equations along (u, v, h) of vertex b
        const double dt_u = ts * ua * kOne3, dt_v = ts * va * kOne3, dt_h = 0.5 * ts * g * kOne3;
        const double dc_u = adt * (kOne3 * ghx + ha * gxb), dc_v = adt * (kOne3 * ghy + ha * gyb),
                     dc_h = A * kOne3 + adv + adt * kOne3 * (gux + gvy);
        const double bs = gih * res * kOne3, buv = bs * ua * va * iw;
        const double dx_u = A * kOne3 + adt * kOne3 * gux + adv + bs * (wmag + ua * ua * iw),
                     dx_v = adt * kOne3 * (guy - cs) + buv,
                     dx_h = adt * g * gxb + kOne3 * (gih * (dres * ua * wmag - bx * ih) + adt * E.wsx * ih * ih);
        const double dy_u = adt * kOne3 * (gvx + cs) + buv, dy_v = A * kOne3 + adt * kOne3 * gvy + adv + bs * (wmag + va * va * iw),
                     dy_h = adt * g * gyb + kOne3 * (gih * (dres * va * wmag - by * ih) + adt * E.wsy * ih * ih);
        // the six scales of the SUPG test functions (continuity: cx, cy; x-momentum: xx, xy; y: yx, yy)
        struct Six { double cx, cy, xx, xy, yx, yy; };
        auto six = [&](double dtau, double du, double dv, double dh, double dc, double dx, double dy) {
            Six s;
            const double dth = dtau * ha + tau * dh;
            s.cx = dtau * (ua * ceq + ha * xeq) + tau * (du * ceq + ua * dc + dh * xeq + ha * dx);
            s.cy = dtau * (va * ceq + ha * yeq) + tau * (dv * ceq + va * dc + dh * yeq + ha * dy);
            s.xx = dth * (g * ceq + ua * xeq) + th * (g * dc + du * xeq + ua * dx);
            s.xy = dth * (va * xeq) + th * (dv * xeq + va * dx);
            s.yx = dth * (ua * yeq) + th * (du * yeq + ua * dy);
            s.yy = dth * (g * ceq + va * yeq) + th * (g * dc + dv * yeq + va * dy);
            return s;
        };
        const Six su = six(dt_u, kOne3, 0., 0., dc_u, dx_u, dy_u), sv = six(dt_v, 0., kOne3, 0., dc_v, dx_v, dy_v),
                  sh = six(dt_h, 0., 0., kOne3, dc_h, dx_h, dy_h);
        // advection of momentum by depth, pressure
        const double guu = k60 * tri(E.u, E.u, Su, Su, Puu, b), guv = k60 * tri(E.u, E.v, Su, Sv, Puv, b),
                     gvv = k60 * tri(E.v, E.v, Sv, Sv, Pvv, b);
        const double pf = kpf * (E.h[b] + Sh), dhd = dt * A * kOne3 * floor_slope(ha, P.dul, eps * kOne3);
        const double frs = kf * dres * kOne3;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double gx = E.gx[a], gy = E.gy[a], w = a == b ? 2.0 : 1.0;
            double* q = o + (3 * a + b) * 9;
            const int f = dflag[a];
            const bool zc = (f & 5) != 0, zm = (f & 6) != 0;
            // continuity
            const double pb = Sh + E.h[b];
            const double cu = k12 * gx * pb + gx * su.cx + gy * su.cy;
            const double cv = k12 * gy * pb + gx * sv.cx + gy * sv.cy;
            const double ch = k12 * (gx * (Su + E.u[b]) + gy * (Sv + E.v[b])) + tc * w + gx * sh.cx + gy * sh.cy;
            // x-momentum
            double xu = tvh * gy + 2. * tuh * gx + kd * (2. * gxb * gx + gyb * gy) + kfr * w * fuu[b] + gx * su.xx + gy * su.xy;
            double xv = tuh * gy + kd * gxb * gy + kfr * w * fuv[b] + gx * sv.xx + gy * sv.xy;
            double xh = guv * gy + guu * gx + dhd * (dxx * gx + dxy * gy) + frs * (sfx + fx[a]) + pf * gx + kb * gzx * w +
                        gx * sh.xx + gy * sh.xy;
            // y-momentum
            double yu = tvh * gx + kd * gyb * gx + kfr * w * fuv[b] + gx * su.yx + gy * su.yy;
            double yv = tuh * gx + 2. * tvh * gy + kd * (gxb * gx + 2. * gyb * gy) + kfr * w * fvv[b] + gx * sv.yx + gy * sv.yy;
            double yh = guv * gx + gvv * gy + dhd * (dxy * gx + dyy * gy) + frs * (sfy + fy[a]) + pf * gy + kb * gzy * w +
                        gx * sh.yx + gy * sh.yy;
            if (a == b) {
                xu += tm * mb;
                yv += tm * mb;
                xh += tm * E.u[a] * ms;
                yh += tm * E.v[a] * ms;
            }
            if (cs != 0.0) {   // sum_bc T_abc h_b v_c and its slopes
                const double T = a == b ? 1.0 : 0.0;
                auto d = [&](double Y, const double* y) { return Y * (1.0 + T) + y[b] + y[a] + 2.0 * T * y[a]; };
                const double dh = kc * d(Sh, E.h);
                xv -= dh;
                yu += dh;
                xh -= kc * d(Sv, E.v);
                yh += kc * d(Su, E.u);
            }
            // pressure on the element's own edges: the two that meet at vertex a
            {
                const int n = (a + 1) % 3, p = (a + 2) % 3;
                const double ny = E.y[n] - E.y[a], nx = E.x[a] - E.x[n];   // edge a -> n, this vertex first
                const double py = E.y[a] - E.y[p], px = E.x[p] - E.x[a];   // edge p -> a, this vertex second
                double sn = 0.0, sp = 0.0;
                if (b == a) {
                    sn = kq * (6. * E.h[a] + 2. * E.h[n]);
                    sp = kq * (6. * E.h[a] + 2. * E.h[p]);
                } else if (b == n) {
                    sn = kq * (2. * E.h[a] + 2. * E.h[n]);
                } else {
                    sp = kq * (2. * E.h[a] + 2. * E.h[p]);
                }
                xh += ny * sn + py * sp;
                yh += nx * sn + px * sp;
            }
            q[0] = zm ? 0.0 : xu;
            q[1] = zm ? 0.0 : xv;
            q[2] = zm ? 0.0 : xh;
            q[3] = zm ? 0.0 : yu;
            q[4] = zm ? 0.0 : yv;
            q[5] = zm ? 0.0 : yh;
            q[6] = zc ? 0.0 : cu;
            q[7] = zc ? 0.0 : cv;
            q[8] = zc ? 0.0 : ch;
        }
    }
}

}  // namespace sw2
