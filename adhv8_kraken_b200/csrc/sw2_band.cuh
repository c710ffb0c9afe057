// sw2_band.cuh -- the exact banded LU solve of one Newton iteration's linear system.
//
// The reference's default linear solver factors the whole Jacobi-scaled system exactly
// (OP BLK 1: one node block, profile LU of solv_blk_set_profile, src/solver/solv_blk_profile.c:5-79,
// applied by solv_blk_solve, src/solver/solv_blk_solve.c:5-62) and runs BiCGSTAB on top of it,
// which then stops at its first test: the solution is LU^-1 b to round-off.  Block-Jacobi
// BiCGSTAB stalls on systems whose time step is many wave-crossings of an element (the QA decks
// the reference ships run at CFL numbers of tens), so a context may ask for this path instead
// (SW2GPU_PREC_BAND): the nodes are renumbered in reverse Cuthill-McKee order on the host, the
// scaled system S A S is scattered into a row-major band of half-width bw (dofs), factored in
// place without pivoting (as the reference's profile LU), and the two triangular solves give the
// increment directly.  A band whose factor window fits in shared memory (bw <= 136) is factored
// in panels of eight pivots (k_band_window); a wider one is walked pivot by pivot from global
// memory (k_band_factor, k_band_solve), the threads sharing each pivot's bw x bw update.  The
// work is n bw^2 for the factor and n bw for a solve, so the path is for the small and medium
// systems of the reference's test decks, not for the 1M-triangle meshes (where the band does not
// fit in the limit sw2gpu_create applies).
#pragma once
#include <cuda_runtime.h>

#include "sw2_krylov.cuh"   // KrylovCtl

namespace sw2 {

constexpr int kBandThreads = 1024;

struct BandArgs {
    int V, n, bw, width;        // nodes, 3V dofs, half-width (dofs), row stride 2 bw + 1
    const int* perm;            // [V] new position of node i
    const int *rowptr, *col;    // BCSR pattern (sorted columns, diagonal included)
    const double* val;          // BCSR values [nnzb][9]
    const double* S;            // Jacobi scale [3V]
    const double* bs;           // scaled right-hand side S R [3V]
    double* band;               // [n][width], a(i, j) at i * width + (j - i + bw)
    double* y;                  // [n] permuted right-hand side, then the solution
};

// a(i, j) of the band (callers keep |i - j| <= bw)
__device__ __forceinline__ double& band_at(const BandArgs& B, int i, int j) {
    return B.band[(size_t)i * B.width + (j - i + B.bw)];
}

// S A S of one BCSR block into the band (thread k: block k of row `row[k]`), the band zeroed before
__global__ void k_band_fill(const __grid_constant__ BandArgs B, const int* __restrict__ blk_row, int nnzb) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nnzb) return;
    const int i = blk_row[k], j = B.col[k];
    const int pi = 3 * B.perm[i], pj = 3 * B.perm[j];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++)
            band_at(B, pi + r, pj + c) = B.val[(size_t)k * 9 + 3 * r + c] * (B.S[3 * i + r] * B.S[3 * j + c]);
}

// the right-hand side in the band's order
__global__ void k_band_rhs(const __grid_constant__ BandArgs B) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.V) return;
#pragma unroll
    for (int r = 0; r < 3; r++) B.y[3 * B.perm[i] + r] = B.bs[3 * i + r];
}

// In-place LU without pivoting, one CTA: for every pivot k the multipliers l(i, k) = a(i, k) /
// a(k, k) of the rows below it within the band, then the rank-1 update a(i, j) -= l(i, k) a(k, j)
// of the trailing bw x bw block.  A zero pivot gives an infinite or NaN solution, which the Newton
// loop's norms report (the reference's profile LU does not pivot either).
__global__ void __launch_bounds__(kBandThreads) k_band_factor(const __grid_constant__ BandArgs B) {
    const int n = B.n, bw = B.bw;
    for (int k = 0; k < n; k++) {
        const int m = min(bw, n - 1 - k);   // rows (and columns) of the trailing block
        const double piv = band_at(B, k, k);
        for (int t = threadIdx.x; t < m; t += blockDim.x) band_at(B, k + 1 + t, k) /= piv;
        __syncthreads();
        for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
            const int i = k + 1 + t / m, j = k + 1 + t % m;
            band_at(B, i, j) -= band_at(B, i, k) * band_at(B, k, j);
        }
        __syncthreads();
    }
}

// Forward (unit lower) and backward (upper) substitution in place in y, one CTA; every step
// updates the rows the pivot reaches within the band.
__global__ void __launch_bounds__(kBandThreads) k_band_solve(const __grid_constant__ BandArgs B) {
    const int n = B.n, bw = B.bw;
    for (int k = 0; k < n; k++) {
        const double yk = B.y[k];
        const int m = min(bw, n - 1 - k);
        for (int t = threadIdx.x; t < m; t += blockDim.x) B.y[k + 1 + t] -= band_at(B, k + 1 + t, k) * yk;
        __syncthreads();
    }
    for (int k = n - 1; k >= 0; k--) {
        if (threadIdx.x == 0) B.y[k] = B.y[k] / band_at(B, k, k);
        __syncthreads();
        const double xk = B.y[k];
        const int m = min(bw, k);
        for (int t = threadIdx.x; t < m; t += blockDim.x) B.y[k - 1 - t] -= band_at(B, k - 1 - t, k) * xk;
        __syncthreads();
    }
}

// ---- the same factorisation in panels, the active window in shared memory ------------------
//
// Bound: the chain of pivots.  Every pivot's division and update wait for the one before, so the
// time is (pivots) x (latency per pivot); the work, n bw^2 products, is small beside it.  The walk
// above pays two block barriers and two trips to L2 per pivot.  Here one CTA keeps the window of
// the band that the next eight pivots touch in shared memory and takes eight pivots at a time:
//   1. one thread per column solves the panel's eight rows of U (and of the right-hand side, which
//      is carried along as one more column, so there is no separate forward substitution);
//   2. the next panel's columns take their rank-8 update;
//   3. one warp factors the next panel (eight columns, the rows they reach) in registers, a pivot's
//      row broadcast by shuffles: no barrier between pivots; meanwhile the other warps update the
//      rest of the trailing block, write the finished rows out and fetch the eight rows and columns
//      that enter the window with cp.async.
// The updates run on the FP64 tensor cores (mma.m8n8k4: eight columns are two of its steps, and it
// needs a quarter of the shared-memory reads that per-element products need).
// Three barriers per eight pivots.  The window is circular: row i and column j live at
// (i mod wm, j mod wm) with wm = bw rounded up to eights plus 24: the panel, the rows it reaches, the
// eight more that the next one reaches and the eight being fetched; its rows are wm + 4 doubles apart, which spreads the fragments' rows over
// the banks.  Rows past n are identity rows.
// The back substitution takes 32 rows at a time: a warp per row for the products with what is
// known, one warp for the 32 x 32 triangle.
// Channel of 1,111 nodes (n = 3333, bw 41) on a B200: 7.9 ms per factor and solve with the kernels
// above, 0.95 ms with this one (2.3 us per eight pivots, of which the panel's chain of eight
// reciprocals, shuffles and products is about 1.1).
constexpr int kBandPanel = 8;
// widest band whose window fits in shared memory (160 rows of 164 doubles, 210 KB of the 227 KB a
// CTA may have); a wider band is walked pivot by pivot in global memory
constexpr int kBandWindowMaxBw = 136;
constexpr int kBandBackRows = 32;
constexpr int kBandWindowThreads = 512;   // 128 registers: the panel warp holds five rows of eight per lane
inline int band_window_rows(int bw) { return (bw + kBandPanel - 1) / kBandPanel * kBandPanel + 3 * kBandPanel; }
inline size_t band_window_smem(int bw) {
    const size_t wm = band_window_rows(bw);
    return sizeof(double) * (wm * (wm + 4) + wm + kBandBackRows * (kBandBackRows + 1) + 2 * kBandBackRows);
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}
// c += a b of one 8 x 8 tile, four products deep
__device__ __forceinline__ void dmma_8x8x4(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// a / b from r = 1 / b correctly rounded: the quotient's remainder corrects it (Markstein, 1990), so
// one reciprocal serves every row of a pivot at the accuracy of a division
__device__ __forceinline__ double div_by(double a, double b, double r) {
    const double q = a * r;
    return __fma_rn(__fma_rn(-b, q, a), r, q);
}

// SLOTS: panel rows per lane (32 SLOTS >= the rows a panel reaches); straight-line code for more
// rows than a narrow band has costs it instruction-cache misses at every panel
template <int SLOTS>
__global__ void __launch_bounds__(kBandWindowThreads) k_band_window(const __grid_constant__ BandArgs B) {
    extern __shared__ __align__(16) double wsm[];
    const int n = B.n, bw = B.bw;
    const int nt = (bw + kBandPanel - 1) / kBandPanel;   // 8-row tiles a panel reaches
    const int wm = (nt + 3) * kBandPanel, ld = wm + 4;
    double* W = wsm;                  // the window
    double* Y = W + wm * ld;          // its right-hand side
    double* T = Y + wm;               // back substitution: the triangle [32][33]
    double* P = T + kBandBackRows * (kBandBackRows + 1);   // reduced right-hand sides [32]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int nwarp = kBandWindowThreads / 32;
    auto wrap = [&](int x) { return x >= wm ? x - wm : x; };   // window position of one below 2 wm
    // window entry of row i, column j (at window row wi, column wj)
    auto entry = [&](int i, int j, int wi, int wj) {
        double* d = W + wi * ld + wj;
        const bool in = i < n && j < n && j - i <= bw && i - j <= bw;
        if (i >= n && i == j) *d = 1.0;
        else cp_async8(d, in ? B.band + (size_t)i * B.width + (j - i + bw) : B.band, in);
    };
    // the eight new indices c0 .. c0 + 7 (at window position wc) against the `len` indices from lo
    // (at wl) up to them and themselves, and their right-hand side, by warps w0, w0 + 1, ...
    auto fetch = [&](int lo, int wl, int c0, int wc, int w0) {
        const int len = c0 - lo;
        for (int r = warp - w0; r < kBandPanel; r += nwarp - w0)          // new rows
            for (int c = lane; c < len + kBandPanel; c += 32) entry(c0 + r, lo + c, wc + r, wrap(wl + c));
        for (int r = 4 * (warp - w0) + (lane >> 3); r < len; r += 4 * (nwarp - w0))   // older rows, new columns
            entry(lo + r, c0 + (lane & 7), wrap(wl + r), wc + (lane & 7));
        if (warp == nwarp - 1 && lane < kBandPanel)
            cp_async8(Y + wc + lane, c0 + lane < n ? B.y + c0 + lane : B.y, c0 + lane < n);
    };
    auto landed = [] { asm volatile("cp.async.wait_all;" ::: "memory"); };
    for (int c = 0; c <= nt; c++) fetch(0, 0, c * kBandPanel, c * kBandPanel, 0);
    landed();
    __syncthreads();
    const int rows = (nt + 1) * kBandPanel;
    // one warp: the panel at window position kb, rows lane + 32 s of its eight columns
    auto factor = [&](int kb) {
        double a[SLOTS][kBandPanel];
        double* w[SLOTS];
#pragma unroll
        for (int s = 0; s < SLOTS; s++) {
            w[s] = W + wrap(kb + min(lane + 32 * s, rows - 1)) * ld + kb;
#pragma unroll
            for (int q = 0; q < kBandPanel; q += 2) {
                const double2 v = *reinterpret_cast<const double2*>(w[s] + q);
                a[s][q] = v.x;
                a[s][q + 1] = v.y;
            }
        }
#pragma unroll
        for (int q = 0; q < kBandPanel; q++) {
            double u[kBandPanel];
#pragma unroll
            for (int c = q; c < kBandPanel; c++) u[c] = __shfl_sync(0xffffffffu, a[0][c], q);
            const double r = 1.0 / u[q];
#pragma unroll
            for (int s = 0; s < SLOTS; s++) {
                const double l = (s > 0 || lane > q) ? div_by(a[s][q], u[q], r) : 0.0;
                if (s > 0 || lane > q) a[s][q] = l;
#pragma unroll
                for (int c = q + 1; c < kBandPanel; c++) a[s][c] = __fma_rn(-l, u[c], a[s][c]);
            }
        }
#pragma unroll
        for (int s = 0; s < SLOTS; s++)
            if (lane + 32 * s < rows) {
#pragma unroll
                for (int q = 0; q < kBandPanel; q += 2)
                    *reinterpret_cast<double2*>(w[s] + q) = make_double2(a[s][q], a[s][q + 1]);
            }
    };
    if (warp == 0) factor(0);
    else fetch(kBandPanel, kBandPanel, rows, rows, 1);
    landed();
    __syncthreads();
    // trailing tiles after the first tile column: `share` warps per tile row (a narrow band has
    // fewer tile rows than there are warps)
    const int share = max(1, (nwarp - 1) / nt), tr0 = (warp - 1) % nt, tp0 = (warp - 1) / nt;
    int kb = 0;   // window position of the panel (a multiple of 8, as wm is: a panel never wraps)
    for (int k0 = 0; k0 < n; k0 += kBandPanel, kb = wrap(kb + kBandPanel)) {
        const int kn = wrap(kb + kBandPanel);   // the next panel's
        // U of the panel's rows: column k0 + 8 + t, or the right-hand side (t = 8 nt)
        if (tid <= kBandPanel * nt) {
            const bool rhs = tid == kBandPanel * nt;
            double* w = rhs ? Y + kb : W + kb * ld + wrap(kn + tid);
            const int step = rhs ? 1 : ld;
            double x[kBandPanel];
#pragma unroll
            for (int q = 0; q < kBandPanel; q++) x[q] = w[q * step];
#pragma unroll
            for (int c = 0; c + 1 < kBandPanel; c++)
#pragma unroll
                for (int q = c + 1; q < kBandPanel; q++) x[q] = __fma_rn(-W[(kb + q) * ld + kb + c], x[c], x[q]);
#pragma unroll
            for (int q = 0; q < kBandPanel; q++) w[q * step] = x[q];
        }
        __syncthreads();
        // trailing block -= L U, tile rows tr: the next panel's columns, then the rest
        auto tile_row = [&](int tr, int tc, int step, int end) {
            const int r0 = wrap(kn + kBandPanel * tr) + (lane >> 2);
            const double* la = W + r0 * ld + kb + (lane & 3);
            const double a0 = -la[0], a1 = -la[4];
            const double* ub = W + (kb + (lane & 3)) * ld + (lane >> 2);
            double* cb = W + r0 * ld + 2 * (lane & 3);
            int c0 = wrap(kn + kBandPanel * tc);
#pragma unroll 2
            for (; tc < end; tc += step, c0 = wrap(c0 + kBandPanel * step)) {
                double2* c = reinterpret_cast<double2*>(cb + c0);
                double2 v = *c;
                dmma_8x8x4(v.x, v.y, a0, ub[c0]);
                dmma_8x8x4(v.x, v.y, a1, ub[4 * ld + c0]);
                *c = v;
            }
        };
        for (int tr = warp; tr < nt; tr += nwarp) tile_row(tr, 0, 1, 1);
        __syncthreads();
        // the next panel by one warp while the others finish this one's update
        if (warp == 0) {
            factor(kn);
        } else {
            fetch(k0 + 2 * kBandPanel, wrap(kn + kBandPanel), k0 + kBandPanel + rows, wrap(kn + rows), 1);
            if (tp0 < share)
                for (int tr = tr0; tr < nt; tr += nwarp - 1) tile_row(tr, 1 + tp0, share, nt);
            // right-hand side of the rows below, and the finished rows of U out to the band: the
            // warps from the other end
            for (int t = kBandWindowThreads - 1 - tid; t < kBandPanel * nt; t += kBandWindowThreads - 32) {
                const int i = wrap(kn + t);
                double y = Y[i];
#pragma unroll
                for (int q = 0; q < kBandPanel; q++) y = __fma_rn(-W[i * ld + kb + q], Y[kb + q], y);
                Y[i] = y;
            }
            for (int q = nwarp - 1 - warp; q < kBandPanel; q += nwarp - 1)
                if (k0 + q < n) {
                    double* out = B.band + (size_t)(k0 + q) * B.width + bw;
                    const double* w = W + (kb + q) * ld;
                    for (int c = q + lane; c < rows; c += 32)
                        if (c - q <= bw && k0 + c < n) out[c - q] = w[wrap(kb + c)];
                    if (lane == 0) B.y[k0 + q] = Y[kb + q];
                }
        }
        landed();
        __syncthreads();
    }
    // back substitution; the window's place now holds the solution of the rows below, x[i] at
    // X[i mod xm].  A warp takes the rows warp and warp + 16 of a block; the block above's
    // operands are loaded while one warp solves this block's triangle.
    double* X = W;
    const int xm = bw + 2 * kBandBackRows;
    for (int t = tid; t < xm; t += kBandWindowThreads) X[t] = 0.0;
    double uv[2][SLOTS], tv[2], yv[2];
    auto operands = [&](int k0, int m) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = warp + nwarp * h;
            const bool live = k0 >= 0 && r < m;
            const double* u = B.band + (size_t)(live ? k0 + r : 0) * B.width + bw;   // u[d]: column i + d
#pragma unroll
            for (int s = 0; s < SLOTS; s++) {
                const int d = m - r + lane + 32 * s;
                uv[h][s] = live && d <= bw && k0 + r + d < n ? __ldcg(u + d) : 0.0;
            }
            // the row's part of the triangle; rows past the end are identity rows
            tv[h] = !live ? (lane == r ? 1.0 : 0.0) : lane >= r && lane < m && lane - r <= bw ? __ldcg(u + lane - r) : 0.0;
            yv[h] = live ? __ldcg(B.y + k0 + r) : 0.0;
        }
    };
    int m = (n - 1) % kBandBackRows + 1, k0 = n - m;   // the short block first: the others are full
    operands(k0, m);
    __syncthreads();
    for (; k0 >= 0; k0 -= kBandBackRows, m = kBandBackRows) {
        const int x1 = (k0 + m) % xm;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = warp + nwarp * h;
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < SLOTS; q++) {
                int xi = x1 + lane + 32 * q;
                if (xi >= xm) xi -= xm;
                if (lane + 32 * q < bw) s = __fma_rn(uv[h][q], X[xi], s);
            }
            T[r * (kBandBackRows + 1) + lane] = tv[h];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) P[r] = yv[h] - s;
        }
        operands(k0 - kBandBackRows, kBandBackRows);
        __syncthreads();
        if (warp == 0) {
            double y = P[lane];
            const double d = T[lane * (kBandBackRows + 1) + lane], rd = 1.0 / d;
#pragma unroll 4
            for (int c = kBandBackRows - 1; c >= 0; c--) {
                const double xc = __shfl_sync(0xffffffffu, div_by(y, d, rd), c);
                if (lane < c) y = __fma_rn(-T[lane * (kBandBackRows + 1) + c], xc, y);
            }
            const double x = div_by(y, d, rd);
            if (lane < m) {
                X[(k0 + lane) % xm] = x;
                B.y[k0 + lane] = x;
            }
        }
        __syncthreads();
    }
}
// the instantiation for a band: the panel's bw + 8 rows (rounded up) in 32 SLOTS
inline void* band_window_kernel(int bw) {
    const int rows = band_window_rows(bw) - 2 * kBandPanel;
    return rows <= 64 ? (void*)k_band_window<2> : rows <= 96 ? (void*)k_band_window<3> : (void*)k_band_window<5>;
}

// The increment in node order, unscaled (x = S y), as the Krylov kernel's exit applies it: the
// state advances by x and sol = -x (fe_sw2_inc, fe_newton.c:561-585), or sol = x for a plain solve;
// the control record reports one converged iteration.
__global__ void k_band_apply(const __grid_constant__ BandArgs B, double* __restrict__ h, double* __restrict__ u,
                             double* __restrict__ v, double* __restrict__ sol, int apply_inc, KrylovCtl* ctl) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        ctl->iterations = 1;
        ctl->converged = 1;
        ctl->rnorm = 0.0;
        ctl->bnorm = 0.0;
    }
    if (i >= B.V) return;
    const int p = 3 * B.perm[i];
    const double x0 = B.y[p] * B.S[3 * i], x1 = B.y[p + 1] * B.S[3 * i + 1], x2 = B.y[p + 2] * B.S[3 * i + 2];
    if (apply_inc) {
        u[i] += x0;
        v[i] += x1;
        h[i] += x2;
        sol[3 * i] = -x0;
        sol[3 * i + 1] = -x1;
        sol[3 * i + 2] = -x2;
    } else {
        sol[3 * i] = x0;
        sol[3 * i + 1] = x1;
        sol[3 * i + 2] = x2;
    }
}

}  // namespace sw2
