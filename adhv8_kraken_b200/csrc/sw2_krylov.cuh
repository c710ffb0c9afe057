// sw2_krylov.cuh -- the linear solve of one Newton iteration as ONE persistent kernel.
//
// Restates solv_bcgstab (src/solver/solv_bcgstab.c:39-301) on the Jacobi-scaled
// system A' = S A S, b' = S R (spv_jacobi), left-preconditioned by M^-1, with the
// reference's stopping test ||r||inf <= atol + rtol ||M^-1 b'||inf and its initial
// guess u = M^-1 b'.  M is the 3x3 block-Jacobi inverse (the reference factors
// OP BLK node blocks exactly; any M that converges gives the same Newton result).
//
// One cooperative launch runs the whole iteration for every instance of a batch: each
// instance owns a contiguous range of CTAs with its own bounded barrier.  Its work is cut
// into a fixed number of virtual CTAs (the grid the instance would get alone); a physical
// CTA runs virtual CTAs pl, pl + np, ... in turn.  Every dot product / norm is a per-virtual-
// CTA partial reduced in the same fixed order by every CTA, so all CTAs of an instance take
// identical control decisions, and an instance's results are bitwise the same alone, in any
// batch and on reruns.  s = r - alpha Ap is never stored: the second sweep forms it from r and Ap.
//
// What bounds it: on large meshes the matrix stream (HBM above about 250k nodes, L2 below), on
// small ones the latency of an iteration's two grid barriers and of the loads behind them.  So
//   - a virtual CTA owns consecutive rows and keeps the vector a sweep multiplies in shared
//     memory, at its own rows and at the rows they refer to (sw2_halo.h): each entry is fetched
//     (and, in the first sweep, updated) once instead of once per neighbour;
//   - an iteration's vector update is part of the next iteration's first sweep, so an iteration
//     is two sweeps and two grid barriers;
//   - the rows are taken in an order with locality, the nodes' own where it has it (sw2_halo.h);
//   - the matrix does not change during a solve, so the copy warp streams its tiles without
//     regard to the barriers, and a CTA whose tiles all fit in its ring fetches them once per solve.
// A batch launch may stop the instances still iterating at an iteration boundary once enough
// CTAs have finished theirs (KrylovTab::done_ctas), keeping the loop scalars in each
// instance's KrylovCtl; the next launch resumes them with all CTAs shared among them.  The
// partial structure stays that of the instance's virtual grid, so the bits do not change.
// On exit the kernel applies the Newton increment: x = S u, state += x (fe_sw2_inc),
// sol = -x (fe_newton.c:561-585).
#pragma once
#include <cuda_runtime.h>

#include <climits>
#include <type_traits>

#include "sw2_halo.h"

namespace sw2 {

// A CTA: 15 row warps (SpMV rows, vector updates, partials) and one copy warp that fills
// the tile ring.  Three warps take a 32-row tile, one thread per component of a row: a thread's
// products need no shuffles and its row's operands, result and dot products are coalesced.  (Eight
// lanes per row in three CTAs of eight warps spent 2,600 cycles on a tile, most of it the latency
// of shuffles and of three-component epilogues on one lane in eight.)  Five groups of three warps:
// with 128 registers a thread nothing spills, and spilled registers are lost from L1 at every barrier
// (six groups 1 to 3 % slower, eight 10 %, four equal on small meshes and 5 % slower on 100k nodes).
// Two forms of the same code: one CTA per SM, the shortest chain between two barriers, while that
// gives every virtual CTA an SM; two per SM (64 registers, shallower rings) for batches and large
// meshes, where an SM would otherwise stand still while its one CTA fills an operand buffer or waits
// (Krylov time of a 256-member ensemble of 5k to 200k triangles, FP64 / mixed: 1,177 / 854 ms with one
// CTA per SM, 859 / 558 with two; 64 members 314 / 221 and 227 / 148; 256 members of 2k to 10k 110
// and 67).  Both compute the same bits.
constexpr int kTileRows = 32;
constexpr int kTileThreads = 3 * kTileRows;
constexpr int kKrylovGroups = 5;                                 // tiles in work at once
constexpr int kKrylovRowThreads = kKrylovGroups * kTileThreads;
constexpr int kKrylovWarps = kKrylovRowThreads / 32;             // warps that hold partials
constexpr int kKrylovThreads = kKrylovRowThreads + 32;
constexpr long long kBarrierSpinLimit = 1ll << 23;   // polls (a few seconds: each is an L2 round trip), then error
constexpr long long kMbarSpinLimit = 1ll << 20;      // polls (about a second) of one tile mbarrier, then error
// polls (of about a microsecond) the copy warp waits for a released stage: longer than any grid
// barrier the row warps may be in (they tell it when they leave)
constexpr long long kCopyIdleLimit = 1ll << 25;
// a launch may bound its waits more tightly (KrylovArgs::spin_limit / copy_limit, 0 = these
// defaults): failure-detection tests make a wait run out that way, without a fault
constexpr int kStall = 40;                           // iterations without a new best residual
static_assert(kTileRows == kHaloTileRows, "tiles of the share tables");
// Second sweeps take the tiles of a virtual CTA from the last to the first: what the first sweep left
// in L2, and the operands of the rows it wrote last, are read again before they are evicted.
constexpr bool kAlternate = true;
// Virtual CTAs of an instance, at most one per SM (fixed: they set the reduction order, so no tuning
// knob may): five tiles each, one per warp group, which is what a CTA of a batch gets through fastest
// (an engine of 12 basins of 5k to 40k triangles: 21.1 ms with five, 25.2 with two, 28.3 with one);
// two tiles each up to 128 tiles, whose solves are launched alone more often and where a tile's own
// time counts (the 4k channel: 11.4 us per iteration with two, 12.0 with five; 7k triangles 13.3 and
// 15.1; from 500 tiles on within 3 %).
// At most one per SM, two from pair_rows rows on (kPairRows): there an iteration is no longer the
// latency of its barriers but the traffic of its sweeps, and two CTAs on an SM fill their operands
// and multiply at different times.
inline int krylov_vgrid(int V, int sms, int pair_rows = INT_MAX) {
    const int nt = (V + kTileRows - 1) / kTileRows;
    const int per = nt <= 128 ? 2 : kKrylovGroups;
    const int v = (nt + per - 1) / per, most = V >= pair_rows ? 2 * sms : sms;
    return v < 1 ? 1 : v > most ? most : v;
}
// Where a mesh on its own gets two virtual CTAs per SM, by measurement (us per iteration, one and
// two): FP64 100k nodes 33.3 and 34.1, 250k 72.6 and 74.1, 500k 145 and 140; mixed 100k 33.0 and 33.7,
// 130k 40.5 and 38.4, 250k 73.2 and 64.0, 2M 570 and 433.
template <typename MT>
constexpr int kPairRows = sizeof(MT) == 4 ? 120000 : 300000;

// Blocks of one launch over a batch: instance ids[j] owns blocks boff[j] .. boff[j+1]-1.
// Passed by value (kernel parameter space), so lookups are uniform constant-bank reads.
constexpr int kMaxBatch = 256;
struct LaunchMap {
    int n;
    int boff[kMaxBatch + 1];
    int ids[kMaxBatch];
};
// instance id of this block; lb = block index inside the instance, nb = its block count
__device__ __forceinline__ int map_block(const LaunchMap& mp, int& lb, int& nb) {
    const int b = blockIdx.x;
    int lo = 0, hi = mp.n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (mp.boff[mid] <= b) lo = mid;
        else hi = mid;
    }
    lb = b - mp.boff[lo];
    nb = mp.boff[lo + 1] - mp.boff[lo];
    return mp.ids[lo];
}

struct KrylovCtl {
    unsigned count;       // barrier arrivals since the launch (zeroed before it)
    unsigned pad0;
    int err;              // 1 = a barrier or tile-copy wait ran out
    int iterations;
    int converged;        // 1 = stopping test met, 0 = hit max_lin_it
    int pad;
    double rnorm, bnorm;
    // A batch launch may pause an instance at the top of an iteration so that a later launch,
    // with the CTAs of the instances that have finished, resumes it (KrylovTab::done_ctas).  The
    // instance's first CTA sets pause_at (the iteration at whose top it stops) before the
    // iteration's second grid barrier; every CTA reads it at the next loop top.  The loop's
    // scalars are kept here; the vectors stay where they are.
    int pause_at;         // 0: no pause requested
    int paused;           // 1: the launch ended at a pause, the solve resumes in the next one
    int s_it, s_best_it, s_pending, s_upd, s_cur, s_nred, s_ucur, pad1;
    double s_rnorm, s_tol, s_rho, s_alpha, s_omega, s_beta, s_best;
};

// Grid barrier with a bounded spin.  Arrivals only ever add to one counter, so the b-th
// barrier of a launch is passed once the counter reaches b * nblocks (`epoch`, per CTA): the
// last arrival releases everyone without a second atomic.  Returns false (and sets ctl->err)
// if any block gave up; the caller then returns, so the kernel always terminates.  The error
// word is read once, by thread 0, and the decision reaches the whole CTA through shared
// memory: another CTA may set the word at any moment, and threads reading it one by one could
// disagree, some returning while the rest of the CTA waits for them at its next barrier.
constexpr int kBarRows = 1;   // named barrier of the Krylov CTA's row warps alone (0 is __syncthreads')
constexpr int kBarPoll = 2;   // of the warps that collect a reduction
__device__ __forceinline__ void bar_sync_n(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_rows() { bar_sync_n(kBarRows, kKrylovRowThreads); }
__device__ __forceinline__ bool grid_sync(KrylovCtl* ctl, unsigned nblocks, unsigned& epoch, long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        epoch += nblocks;
        __threadfence();
        atomicAdd(&ctl->count, 1u);
        // tight bounded poll (acquire loads, no sleep: a wake-up later than the last arrival
        // would be paid at every barrier)
        long long spins = 0;
        for (;;) {
            unsigned cur;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(&ctl->count) : "memory");
            if ((int)(cur - epoch) >= 0) break;
            if (++spins > limit || *(volatile int*)&ctl->err) {
                atomicExch(&ctl->err, 1);
                break;
            }
        }
        // no trailing fence: the acquire load orders this thread's later accesses, and the
        // __syncthreads below orders the rest of the CTA's after it
        s_ok = *(volatile int*)&ctl->err == 0;
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ void bar_arrive_n(int id, int count) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// fixed-order warp tree (xor shuffles): every lane ends with the same value
__device__ __forceinline__ double warp_combine(double a, bool is_max) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xffffffffu, a, o);
        a = is_max ? fmax(a, t) : a + t;
    }
    return a;
}

// ---- reduction and grid barrier in one ----------------------------------------------------------
// Every virtual CTA publishes its partials of a reduction once the sweep's stores of its rows are
// ordered before them; every CTA waits for all partials, which is also the barrier the next sweep
// needs, and combines them in the same fixed order.  Against a counter barrier followed by loads
// of the partials this saves a trip to L2 and the arrivals' queue at one address.  A partial is
// published as two 64-bit words, each half of the value beside the reduction's number, so no word
// is ever seen torn; the top bit of the number says that a tile-copy wait ran out.  Two buffers in
// turn: a slot is rewritten two reductions later, when every CTA has read it.
constexpr unsigned kTagError = 0x80000000u;
constexpr int kMaxVirtual = 320;                     // virtual CTAs of an instance
constexpr size_t krylov_part_doubles(int vgrid) { return (size_t)2 * vgrid * 4 * 2; }
__device__ __forceinline__ void publish(double* slot, double v, unsigned tag) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned long long w0 = (b & 0xffffffff00000000ull) | tag, w1 = (b << 32) | tag;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(slot), "l"(w0), "l"(w1) : "memory");
}
// true when the slot holds reduction `n`; v its value, err whether its CTA flagged an error
__device__ __forceinline__ bool peek(const double* slot, unsigned n, double& v, bool& err) {
    unsigned long long w0, w1;
    asm volatile("ld.acquire.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w0), "=l"(w1) : "l"(slot) : "memory");
    if (((unsigned)w0 & ~kTagError) != n || ((unsigned)w1 & ~kTagError) != n) return false;
    err = ((unsigned)w0 & kTagError) != 0;
    v = __longlong_as_double((long long)((w0 & 0xffffffff00000000ull) | (w1 >> 32)));
    return true;
}

template <typename T>
__device__ __forceinline__ T ldv(const T* p) { return __ldcg(p); }

// three values at once (their shuffles overlap): a summed, b and c summed or maximised (values >= 0)
__device__ __forceinline__ void warp_combine3(double& a, double& b, double& c, bool bmax, bool cmax) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ta = __shfl_xor_sync(0xffffffffu, a, o), tb = __shfl_xor_sync(0xffffffffu, b, o),
                     tc = __shfl_xor_sync(0xffffffffu, c, o);
        a += ta;
        b = bmax ? (tb > b ? tb : b) : b + tb;
        c = cmax ? (tc > c ? tc : c) : c + tc;
    }
}

// max(m, |x|) of m >= 0; a NaN x leaves m, as fmax does
__device__ __forceinline__ double max_abs(double m, double x) {
    x = fabs(x);
    return x > m ? x : m;
}

// inverse of a 3x3 block (cofactors over the determinant); false (and the identity) when
// the block is singular or not finite
__device__ __forceinline__ bool inv3(const double* a, double* out) {
    const double c00 = a[4] * a[8] - a[5] * a[7], c01 = a[5] * a[6] - a[3] * a[8], c02 = a[3] * a[7] - a[4] * a[6];
    const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
    if (det == 0.0 || !isfinite(det)) {
#pragma unroll
        for (int q = 0; q < 9; q++) out[q] = (q % 4 == 0) ? 1.0 : 0.0;
        return false;
    }
    const double id = 1.0 / det;
    out[0] = c00 * id;
    out[1] = (a[2] * a[7] - a[1] * a[8]) * id;
    out[2] = (a[1] * a[5] - a[2] * a[4]) * id;
    out[3] = c01 * id;
    out[4] = (a[0] * a[8] - a[2] * a[6]) * id;
    out[5] = (a[2] * a[3] - a[0] * a[5]) * id;
    out[6] = c02 * id;
    out[7] = (a[1] * a[6] - a[0] * a[7]) * id;
    out[8] = (a[0] * a[4] - a[1] * a[3]) * id;
    return true;
}

// o = d * b for 3x3 blocks (row-major), formed in FP64 and stored as MT
template <typename MT>
__device__ __forceinline__ void fold_block(const double* d, const double* b, MT* o) {
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++)
            o[3 * r + c] = (MT)(d[3 * r] * b[c] + d[3 * r + 1] * b[3 + c] + d[3 * r + 2] * b[6 + c]);
}

struct KrylovArgs {
    int V;
    const int *rowptr, *col;  // off-diagonal block structure of the folded operator M^-1 A'
    // staged sweeps (sw2_halo.h): sub-ranges per virtual CTA and their halo rows
    int nsub;
    const int *hptr, *hidx;
    // node of each row when the solve takes the rows in another order than the nodes (null: row i is
    // node i); S, bs, Dinv, the state and sol are in node order, everything else in row order
    const int* order;
    // tile records (TileRecord): where record m and its blocks begin, in 16-byte units from A;
    // null: A holds the blocks in pattern order alone (direct sweeps only)
    const int *toff, *boff;
    const double* S;          // scale vector [3V]
    const double* bs;         // scaled rhs S R [3V]
    double atol;              // absolute Krylov tolerance (the relative one is per launch)
    int maxit;
    double *h, *u, *v;        // state, incremented on exit
    double* sol;              // -x on exit (x itself when apply_inc == 0)
    int apply_inc;            // 1: Newton increment of the state; 0: plain solve
    double* part;             // [2][vgrid][4] published partials (krylov_part_doubles), zeroed before the solve
    KrylovCtl* ctl;
    int vgrid;                // virtual CTAs: the partial structure, fixed per instance
    long long spin_limit;     // polls of a grid-barrier wait before it gives up (0: kBarrierSpinLimit)
    long long copy_limit;     // polls of a tile-copy wait before it gives up (0: kMbarSpinLimit)
};

// one instance of a Krylov launch
struct KrylovInst {
    KrylovArgs K;
    const void* A;            // folded off-diagonal blocks, MT
    const double* Dinv;       // FP64 block-Jacobi inverses (b = M^-1 b' only)
    double* vec[10];          // two copies of u, q, As, and two copies of r, p, Ap
};
constexpr int kKrylovVectors = 10;

// The folded operator is stored as one record per tile of kTileRows rows, so that one bulk copy
// brings a tile up (three, for blocks, columns and row pointers, took the issuing lane as long as the
// tile takes from HBM): its row pointers relative to the tile, its blocks' columns in the sub-range's
// operand buffer (sw2_halo.h), both 16-bit and written once per mesh, then its blocks, rewritten by
// every solve.  All three start on 16-byte boundaries.
constexpr int kTileHead = 80;   // kTileRows + 1 row pointers, rounded up
__host__ __device__ constexpr int tile_head(int nb) { return kTileHead + ((2 * nb + 15) & ~15); }
__host__ __device__ constexpr long long tile_bytes(int nb, int esz) { return tile_head(nb) + ((9ll * nb * esz + 15) & ~15ll); }
// the mesh's part of every tile record: one warp per tile
static __global__ void k_tile_heads(int V, const int* __restrict__ rowptr, const unsigned short* __restrict__ lcol,
                                    const int* __restrict__ toff, unsigned char* __restrict__ rec) {
    const int m = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
    if (m * kTileRows >= V) return;
    unsigned short* h = reinterpret_cast<unsigned short*>(rec + 16 * (size_t)toff[m]);
    const int k0 = rowptr[m * kTileRows], k1 = rowptr[min(V, (m + 1) * kTileRows)];
    for (int r = lane; r <= kTileRows; r += 32) h[r] = (unsigned short)(rowptr[min(V, m * kTileRows + r)] - k0);
    for (int k = lane; k < k1 - k0; k += 32) h[kTileHead / 2 + k] = lcol[k0 + k];
}

// Shared memory of the staged sweeps: the operand buffer, then the ring of tile records.
struct StageLayout {
    unsigned stage_bytes, x_bytes;
};
__host__ __device__ constexpr unsigned stage_x_bytes(int rows) { return ((unsigned)rows * 24u + 127u) & ~127u; }
// the largest operand buffer (24 KB): with two CTAs on an SM what is left beside a ring of five tiles
// each; the 1,700 rows a virtual CTA of the 1M-triangle basin has and their halo in two sub-ranges.
// (Twice as much fits with one CTA per SM; that is 4 % faster on FP64 meshes of about 250k nodes alone,
// 70.0 against 72.6 us per iteration, but a batch with such a member could not share its SMs.)
constexpr int kHaloCapRows = 1024;
constexpr int kHaloKeep = 1024;   // halo rows whose numbers a CTA with one sub-range keeps in shared memory

// Where a Krylov launch finds its instances.  KrylovOne: one instance, its record and
// tolerance kernel parameters; KrylovTab: a batch, records in a device table, the map and
// each mapped instance's relative tolerance in the parameters.
struct KrylovOne {
    static constexpr bool kInTable = false;
    KrylovInst Q;
    double rtol;
    const double* rtol_dev;   // when set, the tolerance is read here (a launch replayed from a
                              // CUDA graph takes each Newton iteration's tolerance from memory)
    StageLayout lay;
    __device__ __forceinline__ const KrylovInst& get(int& pl, int& np, double& rt) const {
        pl = blockIdx.x;
        np = gridDim.x;
        rt = rtol_dev ? __ldcg(rtol_dev) : rtol;
        return Q;
    }
    __device__ __forceinline__ unsigned* done_counter() const { return nullptr; }
    __device__ __forceinline__ unsigned pause_threshold() const { return 0u; }
    __device__ __forceinline__ bool resuming() const { return false; }
};
struct KrylovTab {
    static constexpr bool kInTable = true;
    const KrylovInst* tab;
    LaunchMap mp;
    double rtol[kMaxBatch];
    StageLayout lay;
    const double* rtol_dev;   // when set, instance k's tolerance is read at rtol_dev[k] (graph replays)
    // Rebalancing (host-driven launches only): every CTA whose instance finished adds one to
    // *done_ctas (zeroed before the launch); once it reaches pause_after, the instances still
    // running pause at their next iteration top.  resume = 1: every instance of the launch
    // continues a paused solve from the scalars in its KrylovCtl.  An instance's partial
    // structure depends on its virtual grid alone, so its bits do not depend on where it paused
    // nor on how many CTAs each launch gave it.
    unsigned* done_ctas;      // nullptr: no pausing
    unsigned pause_after;
    int resume;
    __device__ __forceinline__ unsigned* done_counter() const { return done_ctas; }
    __device__ __forceinline__ unsigned pause_threshold() const { return pause_after; }
    __device__ __forceinline__ bool resuming() const { return resume != 0; }
    __device__ __forceinline__ const KrylovInst& get(int& pl, int& np, double& rt) const {
        int nb;
        const int b = blockIdx.x;
        int lo = 0, hi = mp.n;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (mp.boff[mid] <= b) lo = mid;
            else hi = mid;
        }
        pl = b - mp.boff[lo];
        nb = mp.boff[lo + 1] - mp.boff[lo];
        np = nb;
        rt = rtol_dev ? __ldcg(rtol_dev + mp.ids[lo]) : rtol[lo];
        return tab[mp.ids[lo]];
    }
};

// the control words of the instances a launch resumes: a fresh barrier, no pause pending (the
// saved scalars stay)
static __global__ void k_krylov_rearm(KrylovCtl* ctl, const __grid_constant__ LaunchMap mp) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= mp.n) return;
    KrylovCtl* c = ctl + mp.ids[j];
    c->count = 0;
    c->pause_at = 0;
    c->paused = 0;
}

// ---- tile staging: one bulk copy per tile, completion on an mbarrier -------------------------
// Tile m = rows [m kTileRows, (m+1) kTileRows) of the solve; its record begins and ends on 16-byte
// boundaries (the bulk-copy rule).
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// bulk copy with an L2 eviction policy
__device__ __forceinline__ void bulk_load_hint(void* dst, const void* src, unsigned bytes, unsigned long long* bar,
                                               unsigned long long policy) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
        : "memory");
}
// eviction policy of the matrix stream.  A matrix that the L2 (126 MB) can hold beside the vectors
// stays in it; a larger one passes through first-out, which keeps the vectors in (1M triangles, a
// matrix of 222 MB: 136 us per iteration, 147 without the hint; 200k, 45 MB: 31.7 with it, 30.7
// without; 260k mixed, 31 MB: 39.1 and 37.9).
constexpr long long kStreamFirstOutBytes = 64ll << 20;
__device__ __forceinline__ unsigned long long policy_stream(bool first_out) {
    unsigned long long p;
    if (!first_out) {
        asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
        return p;
    }
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// bounded wait (at most `limit` polls) for the completion of the phase with the given parity.
// A try_wait poll may itself suspend the thread for a hardware time window, long enough for a
// tile copy to land; a limit below kShortWait polls with the non-blocking test_wait instead, so
// that a short limit really bounds the wait (failure-detection tests).
constexpr long long kShortWait = 64;
constexpr unsigned kWaitHintNs = 1000;
// one poll that may suspend for the hint's time
__device__ __forceinline__ bool mbar_poll(unsigned long long* bar, unsigned parity) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity), "r"(kWaitHintNs)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, long long limit) {
    const unsigned a = smem_addr(bar);
    if (limit < kShortWait) {
#pragma unroll 1
        for (long long k = 0; k < limit; k++) {
            unsigned done;
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(done)
                : "r"(a), "r"(parity)
                : "memory");
            if (done) return true;
        }
        return false;
    }
#pragma unroll 1
    for (long long k = 0; k < limit; k++) {
        // the suspend-time hint (ns) caps how long one poll may park the thread, so `limit` polls
        // bound the wait to about limit microseconds; a completed phase wakes the thread at once
        if (mbar_poll(bar, parity)) return true;
    }
    return false;
}

// explicit fused multiply-add, a * b + c rounded once (the library is built without implicit
// contraction so that every kernel instantiation rounds alike; hot loops state their FMAs)
__device__ __forceinline__ double fmadd(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fmadd(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// Off-diagonal row sum y = sum_j (B_ij x_j)_c of the folded operator (B_ij = D_i^-1 A'_ij, blocks
// kb..ke-1) for component c of a node row, with x_j from gat(j, x); the caller adds the identity
// diagonal block's x_i.  blk(k) / cix(k) give block k's values and column (from the staged tile in
// shared memory, or from global memory).  Products and sums are formed in the matrix type MT (FP32
// accumulation on the mixed path), one running sum per column of the blocks in block order, so
// staged and direct sweeps give bitwise identical results.
template <typename MT, typename VT, class BLK, class CIX, class GAT>
__device__ __forceinline__ VT row_apply(int c, int kb, int ke, BLK blk, CIX cix, GAT gat) {
    MT a0 = 0, a1 = 0, a2 = 0;
#pragma unroll 2
    for (int k = kb; k < ke; k++) {
        const MT* bk = blk(k) + 3 * c;
        const MT m0 = bk[0], m1 = bk[1], m2 = bk[2];
        VT x[3];
        gat(cix(k), x);
        a0 = fmadd(m0, (MT)x[0], a0);
        a1 = fmadd(m1, (MT)x[1], a1);
        a2 = fmadd(m2, (MT)x[2], a2);
    }
    return (VT)((a0 + a1) + a2);
}

// MT: matrix storage and SpMV accumulation type; VT: Krylov vector type (FP64 on both paths:
// FP32 vectors let the recursively updated residual drift away from the true one and the
// iteration stagnates).  Per instance, A holds the folded off-diagonal blocks D_i^-1 A'_ij
// (rowptr / col of K) and Dinv the FP64 inverses (used once, for b = M^-1 b').
// STAGES > 0: the row warps read the operand from the buffer in shared memory and the matrix from
// a ring of STAGES - 1 tiles per warp group filled by bulk copies of the copy warp (completion on an
// mbarrier per tile, release on another); the operands of large matrices' rows stay in L2
// (policy_stream).  PER_SM: CTAs that share an SM.  STAGES = 0: the threads load blocks and operands from global memory (meshes
// whose tiles or halos do not fit).  Every variant computes the same bits.
//
// Measured (B200, us per iteration, with eight lanes per row, operands gathered from L2, three copies
// per tile and a counter barrier before): 4k-triangle channel 12.6 -> 11.1, 32k mixed 24 -> 16.8, 200k
// 52 -> 33.3, 260k mixed 59 -> 38.4, 1M 140 -> 140, 4M mixed 492 -> 433.  An iteration of the 1M basin
// moves 444 MB of matrix and 156 MB of vectors (92 us at the measured copy rate); one of the 200k basin
// spends half its time in the latency of its two sweeps' chains: operands, products, sums, fence, poll.
// Entries are numbered in 32 bits: 64-bit indices cost the two-CTA form spills (batches 3 % slower) and
// both the extra instructions (200k 34.9 -> 33.3).
// STAGES of direct sweeps over a pattern without share tables
constexpr int kStagesWhole = -1;
// places of a warp group's ring with two CTAs per SM
template <typename MT>
__host__ __device__ constexpr int pair_places() { return sizeof(MT) == 4 ? 2 : 1; }
// what the row warps do next, and the scalars it takes
enum KrylovNext : int { kSweepInit, kSweepPlain, kSweepUpdate, kSweepS, kSweepEnd, kSweepPause, kSweepFail };
struct KrylovState {
    double rnorm, tol, rho, alpha, omega, beta, best;
    int it, best_it, pending, cur, ucur, next;
    unsigned nred;   // reductions so far: their number, and the buffer in turn
};

template <typename MT, typename VT, int STAGES, int PER_SM, class KS>
__global__ void __launch_bounds__(kKrylovThreads, PER_SM) k_bicgstab(const __grid_constant__ KS src) {
    __shared__ double red[3 * kKrylovWarps];    // a virtual CTA's sums, per warp
    __shared__ KrylovState C;                   // the solve's scalars and the next sweep
    __shared__ int s_hidx[STAGES > 0 ? kHaloKeep : 1];   // the halo rows of a CTA with one sub-range
    __shared__ double s_poll[4 * kKrylovWarps];   // the polling warps' sums and error
    __shared__ int s_stop;                      // the row warps have left
    __shared__ int s_go;                        // a tile wait ran out (a held-back first copy may go)
    constexpr bool STAGED = STAGES > 0;
    // the ring: S places for each group (its tile in work is the launch variant's first stage), so that a place's waits come from one group in order (a parity
    // tells a phase from its neighbours only)
    constexpr unsigned S = STAGED ? STAGES - 1 : 1;
    constexpr int NST = (int)S * kKrylovGroups;
    __shared__ unsigned long long bar[NST];     // per ring tile: its copy has landed ("full")
    __shared__ unsigned long long ebar[NST];    // per ring tile: its three warps are done with it ("empty")
    extern __shared__ __align__(128) unsigned char stage_mem[];
    int pl, np;   // this CTA's index among the instance's np CTAs
    double rtol;
    const KrylovInst& found = src.get(pl, np, rtol);
    // a batch's record is in global memory: a copy the CTA can read at any time
    __shared__ __align__(16) unsigned char s_inst[KS::kInTable ? sizeof(KrylovInst) : 16];
    if (KS::kInTable) {
        for (int k = threadIdx.x; k < (int)(sizeof(KrylovInst) / 4); k += kKrylovThreads)
            reinterpret_cast<int*>(s_inst)[k] = reinterpret_cast<const int*>(&found)[k];
        __syncthreads();
    }
    const KrylovInst& KI = KS::kInTable ? *reinterpret_cast<const KrylovInst*>(s_inst) : found;
    const StageLayout& L = src.lay;
    const KrylovArgs& K = KI.K;
    VT* const xs = reinterpret_cast<VT*>(stage_mem);   // the operand buffer
    unsigned char* const ring = stage_mem + L.x_bytes;
    const int V = K.V;
    const int VG = K.vgrid;
    const int ntiles = (V + kTileRows - 1) / kTileRows;   // >= VG: every virtual CTA has a tile
    auto tile0 = [&](int v) { return (int)((long long)v * ntiles / VG); };
    KrylovCtl* ctl = K.ctl;
    const long long bar_limit = K.spin_limit > 0 ? K.spin_limit : kBarrierSpinLimit;
    const long long copy_limit = K.copy_limit > 0 ? K.copy_limit : kMbarSpinLimit;
    int ntot = 0;   // tiles of this CTA in a sweep; if they all fit in the ring they stay there
#pragma unroll 1
    for (int v = pl; v < VG; v += np) ntot += tile0(v + 1) - tile0(v);
    if (threadIdx.x == 0) {
        s_stop = s_go = 0;
        if (STAGED) {
#pragma unroll 1
            for (int s = 0; s < NST; s++) {
                mbar_init(&bar[s], 1);
                mbar_init(&ebar[s], kTileThreads / 32);
            }
            mbar_init_fence();
        }
    }
    __syncthreads();
    const bool resident = STAGED && ntot <= NST;
    const int hp0 = STAGED && K.nsub == 1 ? __ldg(K.hptr + pl) : 0, nhalo = STAGED && K.nsub == 1 ? __ldg(K.hptr + pl + 1) - hp0 : 0;
    const bool single = STAGED && K.nsub == 1 && pl + np >= VG && nhalo <= kHaloKeep;
    if (single && threadIdx.x < kKrylovRowThreads)   // read after the row warps' first barrier
        for (int h = threadIdx.x; h < nhalo; h += kKrylovRowThreads) s_hidx[h] = __ldg(K.hidx + hp0 + h);

    // ---- the copy warp streams the tiles of sweep after sweep, up to NST ahead of the row warps,
    // until they leave.  Its lanes hold the record offsets of the next 31 tiles (a tile's own loads in
    // front of its copy would be a trip to L2 per tile), its first lane waits and issues.  Every wait
    // is bounded; before it leaves, the copies it issued have landed in the CTA's shared memory.
    if (threadIdx.x >= kKrylovRowThreads) {
        if (!STAGED) return;
        const int lane = threadIdx.x & 31;
        const bool issuer = lane == 0;
        const unsigned long long pol = policy_stream(16ll * __ldg(K.toff + ntiles) > kStreamFirstOutBytes);
        auto stopped = [&] { return *(volatile int*)&s_stop != 0; };
        // a launch with a copy limit so short that it polls without suspending (failure detection)
        // holds its first copy back until a row warp's wait has run out
        if (issuer && copy_limit < kShortWait)
#pragma unroll 1
            for (long long k = 0; k < kCopyIdleLimit && !stopped() && *(volatile int*)&s_go == 0; k++) __nanosleep(100);
        unsigned mine = 0;   // lane g: tiles issued for group g
        unsigned index = 0;  // resident: the tile's own place
        int sweeps = src.resuming() ? 1 : 0;   // a resumed solve goes on with an updating sweep
        const int nsub = K.nsub;
        bool go = true;
#pragma unroll 1
        while (go) {
            const bool back = kAlternate && sweeps >= 2 && sweeps % 2 == 0;   // the sweeps of mode kSweepS
#pragma unroll 1
            for (int v = pl; go && v < VG; v += np) {
                const int ta = tile0(v), nt = tile0(v + 1) - ta;
#pragma unroll 1
                for (int sq = 0; go && sq < nsub; sq++) {
                    const int sb = back ? nsub - 1 - sq : sq;
                    const int m0 = ta + sb * nt / nsub, m1 = ta + (sb + 1) * nt / nsub;
                    // the lowest of the 31 tiles at positions p .. p + 30 of the sub-range, and their offsets
                    auto lowest = [&](int p) { return back ? max(m0, m1 - p - 31) : min(m0 + p, ntiles); };
                    auto offsets = [&](int p) { return __ldg(K.toff + min(lowest(p) + lane, ntiles)); };
                    int next = offsets(0);
#pragma unroll 1
                    for (int p0 = 0; go && p0 < m1 - m0; p0 += 31) {
                        const int here = next, lo = lowest(p0);   // record lo + j: lanes j, j + 1
                        next = offsets(p0 + 31);
#pragma unroll 1
                        for (int p = p0; go && p < p0 + 31 && p < m1 - m0; p++) {
                            const int j = (back ? m1 - 1 - p : m0 + p) - lo, g = p % kKrylovGroups;
                            const int o0 = __shfl_sync(0xffffffffu, here, j), o1 = __shfl_sync(0xffffffffu, here, j + 1);
                            const unsigned n = __shfl_sync(0xffffffffu, mine, g);   // tiles the group has had
                            const unsigned place = resident ? index : (unsigned)g * S + n % S;
                            bool ok = true;
                            if (issuer) {
                                if (!resident && n >= S) {
                                    // the place's previous tile: released by the group's three warps
                                    const unsigned par = (n / S - 1u) & 1u;
                                    long long k = 0;
#pragma unroll 1
                                    while (!mbar_poll(&ebar[place], par) && ++k < kCopyIdleLimit && !stopped()) {}
                                    ok = k < kCopyIdleLimit && !stopped();
                                }
                                if (ok) {
                                    const unsigned bytes = 16u * (unsigned)(o1 - o0);
                                    mbar_arrive_expect_tx(&bar[place], bytes);
                                    bulk_load_hint(ring + place * L.stage_bytes, (const unsigned char*)KI.A + 16 * (size_t)o0, bytes, &bar[place], pol);
                                }
                            }
                            go = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                            if (go && lane == g) mine++;
                            index++;
                        }
                    }
                }
            }
            if (resident || __shfl_sync(0xffffffffu, (int)stopped(), 0)) go = false;
            sweeps++;
        }
        // the last copy into every place has landed before the warp leaves
#pragma unroll 1
        for (int g = 0; g < kKrylovGroups; g++) {
            const unsigned n = __shfl_sync(0xffffffffu, mine, g);
            if (issuer && !resident)
#pragma unroll 1
                for (unsigned i = n > S ? n - S : 0u; i < n; i++) mbar_wait(&bar[(unsigned)g * S + i % S], (i / S) & 1u, kMbarSpinLimit);
        }
        if (issuer && resident)
#pragma unroll 1
            for (unsigned i = 0; i < index; i++) mbar_wait(&bar[i], 0u, kMbarSpinLimit);
        return;
    }

    // ---- the row warps
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = tid / kTileThreads, gt = tid % kTileThreads;   // this thread's tile, entry of it
    const int li = gt / 3, comp = gt % 3;                            // row of the tile, component
    VT* const q = KI.vec[2];
    VT* const As = KI.vec[3];
    // r, p, Ap in two copies (vec[4..5], [6..7], [8..9]): the sweep that applies an iteration's
    // update reads the old copy (at neighbour rows too) and writes the new one
    const int ta0 = tile0(pl), nt0 = tile0(pl + 1) - ta0;
    unsigned tc = 0;     // tiles this group has taken: its place tc % S, mbarrier parity (tc / S) & 1
    bool wait_failed = false;
    using V2 = typename std::conditional<sizeof(VT) == 8, double2, float2>::type;
    auto ld2 = [](const VT* p, unsigned k) { return __ldcg(reinterpret_cast<const V2*>(p + k)); };
    auto st2 = [](VT* p, unsigned k, V2 v) { *reinterpret_cast<V2*>(p + k) = v; };
    if (tid == 0) {
        C.next = kSweepInit;
        if (src.resuming()) {   // the scalars of the paused solve (written by the previous launch)
            C.rnorm = ctl->s_rnorm;
            C.tol = ctl->s_tol;
            C.rho = ctl->s_rho;
            C.alpha = ctl->s_alpha;
            C.omega = ctl->s_omega;
            C.beta = ctl->s_beta;
            C.best = ctl->s_best;
            C.it = ctl->s_it;
            C.best_it = ctl->s_best_it;
            C.pending = ctl->s_pending;
            C.cur = ctl->s_cur;
            C.ucur = ctl->s_ucur;
            C.nred = (unsigned)ctl->s_nred;
            C.next = ctl->s_upd ? kSweepUpdate : kSweepPlain;
        } else {
            C.it = C.best_it = C.cur = C.ucur = 0;
            C.pending = 1;
            C.nred = 0;
            C.beta = 0.0;
            C.alpha = C.omega = 1.0;
        }
    }
    bar_rows();

    // An iteration is two sweeps: Ap = M^-1 A p (first applying the last iteration's update,
    // u += alpha p + omega s, r = s - omega As, p = beta (p - omega Ap) + r, while it brings its operand
    // p up: at its own rows into the other copy, at the halo rows into the operand buffer alone, with
    // the same arithmetic), and As = M^-1 A s with s = r - alpha Ap.  The stopping test of the updated
    // residual follows the first sweep; when it stops the solve, the product that sweep formed is
    // not used.  All sweeps run the same code: an iteration's instructions have to stay in the
    // instruction caches, and what a barrier's fence drops from L1 must not include spilled registers.
#pragma unroll 1
    for (;;) {
        const int mode = C.next;
        if (mode >= kSweepEnd) break;
        const int cur = C.cur;
        const VT al = (VT)C.alpha, om = (VT)C.omega, be = (VT)C.beta;
        const VT* const ro = KI.vec[4 + cur];
        const VT* const po = KI.vec[6 + cur];
        const VT* const apo = KI.vec[8 + cur];
        // the updated p and r of an entry
        auto newp = [&](VT ap, VT p, VT r, VT as, VT& rk) {
            const VT s = fmadd(-al, ap, r);
            rk = fmadd(-om, as, s);
            return fmadd(fmadd(-om, ap, p), be, rk);
        };
        auto newu = [&](VT u, VT ap, VT p, VT r) { return fmadd(om, fmadd(-al, ap, r), fmadd(al, p, u)); };
        // the sweep's operand at entry e
        auto operand = [&](unsigned e) -> VT {
            if (mode == kSweepUpdate) {
                VT rk;
                return newp(ldv(apo + e), ldv(po + e), ldv(ro + e), ldv(As + e), rk);
            }
            if (mode == kSweepS) return fmadd(-al, ldv(apo + e), ldv(ro + e));
            if (mode == kSweepPlain) return ldv(po + e);
            const unsigned r = e / 3, i = K.order ? __ldg(K.order + r) : r;   // b = M^-1 b': row e - 3 r of node i's inverse
            const double* d = KI.Dinv + 9 * (size_t)i + 3 * (e - 3 * r);
            const double* b = K.bs + 3 * (size_t)i;
            return (VT)(d[0] * b[0] + d[1] * b[1] + d[2] * b[2]);
        };
        // first sweep: q . Ap (sum), max |r|; second: As . s, As . As, As . q (sums); at the start:
        // r . r (sum), max |r|, max |b|
        double v0 = 0.0, v1 = 0.0, v2 = 0.0;
        unsigned seen = 0;      // tiles of the virtual CTAs before
        const bool back = kAlternate && mode == kSweepS;
#pragma unroll 1
        for (int v = pl; v < VG; v += np) {
            // a CTA's first virtual CTA has its tiles at hand (the quotients of 64 bits take longer
            // than a small share's products)
            const int ta = v == pl ? ta0 : tile0(v), nt = v == pl ? nt0 : tile0(v + 1) - ta;
            // without staging too: the sub-ranges set the order of the sums
            const int nsub = STAGES == kStagesWhole ? 1 : max(K.nsub, 1);
#pragma unroll 1
            for (int sq = 0; sq < nsub; sq++) {
                const int sb = back ? nsub - 1 - sq : sq;
                const int ma = nsub == 1 ? ta : ta + sb * nt / nsub, mb = nsub == 1 ? ta + nt : ta + (sb + 1) * nt / nsub;
                if (mb == ma) continue;
                const int r0 = ma * kTileRows, n3 = 3 * (min(V, mb * kTileRows) - r0);
                const unsigned base = 3u * (unsigned)r0;   // a multiple of 96: pairs are 16-byte aligned
                // q one tile ahead: its trip to L2 passes under the operand's, then under a tile's products
                auto load_q = [&](int m) {
                    return mode != kSweepInit && m >= ma && m < mb && m * kTileRows + li < V ? ldv(q + (unsigned)(m * kTileThreads + gt)) : (VT)0;
                };
                const int first = back ? mb - 1 - group : ma + group, step = back ? -kKrylovGroups : kKrylovGroups;
                VT qnext = load_q(first);
                if (sq > 0) bar_rows();   // the buffer has been read
                // the operand at the sub-range's own rows
                if (mode == kSweepUpdate) {
                    VT* const rn = KI.vec[5 - cur];
                    VT* const pn = KI.vec[7 - cur];
                    const int n2 = (n3 + 1) / 2;   // the last pair of an odd count: its second entry is padding
                    // the iterate goes to its other copy when the one it comes from is the best so far
                    const VT* const uo = KI.vec[C.ucur];
                    VT* const un = KI.vec[C.ucur ^ C.pending];
#pragma unroll 1
                    for (int k = tid; k < n2; k += kKrylovRowThreads) {
                        const unsigned e = base + 2u * (unsigned)k;
                        const V2 a = ld2(apo, e), p = ld2(po, e), r = ld2(ro, e), s = ld2(As, e), u = ld2(uo, e);
                        V2 uk, rk, pk;
                        uk.x = newu(u.x, a.x, p.x, r.x);
                        uk.y = newu(u.y, a.y, p.y, r.y);
                        pk.x = newp(a.x, p.x, r.x, s.x, rk.x);
                        pk.y = newp(a.y, p.y, r.y, s.y, rk.y);
                        st2(un, e, uk);
                        st2(rn, e, rk);
                        st2(pn, e, pk);
                        v1 = max_abs(v1, (double)rk.x);
                        if (STAGED) xs[2 * k] = pk.x;
                        if (2 * k + 1 < n3) {
                            v1 = max_abs(v1, (double)rk.y);
                            if (STAGED) xs[2 * k + 1] = pk.y;
                        }
                    }
                } else if (STAGED || mode == kSweepInit) {
#pragma unroll 2
                    for (int k = tid; k < n3; k += kKrylovRowThreads) {
                        const VT x = operand(base + k);
                        if (mode == kSweepInit) KI.vec[0][base + k] = x;
                        if (STAGED) xs[k] = x;
                    }
                }
                if (STAGED) {   // and at its halo, from the last thread down: the first ones have the own entries of a small share
                    const int h0 = single ? 0 : __ldg(K.hptr + v * nsub + sb);
                    const int nh = 3 * (single ? nhalo : __ldg(K.hptr + v * nsub + sb + 1) - h0);
#pragma unroll 1
                    for (int t = kKrylovRowThreads - 1 - tid; t < nh; t += kKrylovRowThreads) {
                        const int h = t / 3, j = single ? s_hidx[h] : __ldg(K.hidx + h0 + h);
                        xs[n3 + t] = operand((unsigned)(j * 3 + (t - 3 * h)));
                    }
                }
                bar_rows();
#pragma unroll 1
                for (int m = first; m >= ma && m < mb; m += step) {
                    const int i = m * kTileRows + li;
                    const bool act = i < V;
                    const unsigned e = (unsigned)(m * kTileThreads + gt);   // = 3 i + comp
                    const VT qe = qnext;
                    qnext = load_q(m + step);
                    VT y = 0, x = 0;
                    if (STAGED) {
                        // the tile's place: the group's next one, or its own for good
                        const unsigned place = resident ? seen + (unsigned)(m - ta) : (unsigned)group * S + tc % S;
                        const unsigned par = resident ? 0u : (tc / S) & 1u;
                        const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar[place], par, wait_failed ? kMbarSpinLimit : copy_limit));
                        if (!ok && !wait_failed) {
                            // this warp reads no tile from now on (its rows count as absent), still
                            // waiting, with the default bound, for and releasing every tile, so that the
                            // ring stays in step; the reduction that follows carries the error to every CTA
                            wait_failed = true;
                            if (lane == 0) {
                                atomicExch(&ctl->err, 1);
                                *(volatile int*)&s_go = 1;
                            }
                            __syncwarp();
                            (void)mbar_wait(&bar[place], par, kMbarSpinLimit);
                        }
                        if (act && !wait_failed) {
                            const unsigned char* st = ring + place * L.stage_bytes;
                            const unsigned short* sR = (const unsigned short*)st;
                            const unsigned short* sC = (const unsigned short*)(st + kTileHead);
                            const MT* sA = (const MT*)(st + tile_head(sR[kTileRows]));
                            y = row_apply<MT, VT>(
                                comp, sR[li], sR[li + 1], [&](int k) { return sA + 9 * k; },
                                [&](int k) { return (int)sC[k]; },
                                [&](int j, VT(&xj)[3]) {
#pragma unroll
                                    for (int c = 0; c < 3; c++) xj[c] = xs[3 * j + c];
                                });
                            x = xs[e - base];
                        }
                        if (!resident) {
                            // this warp is done with the tile: one arrival per warp releases it
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&ebar[place]);
                            tc++;
                        }
                    } else if (act) {
                        // the tile's blocks, counted from block 0 of the pattern
                        const MT* At = K.boff ? (const MT*)((const unsigned char*)KI.A + 16 * (size_t)__ldg(K.boff + m)) -
                                                    (size_t)__ldg(K.rowptr + m * kTileRows) * 9
                                              : (const MT*)KI.A;
                        y = row_apply<MT, VT>(
                            comp, __ldg(K.rowptr + i), __ldg(K.rowptr + i + 1), [&](int k) { return At + (size_t)k * 9; },
                            [&](int k) { return __ldg(K.col + k); },
                            [&](int j, VT(&xj)[3]) {
#pragma unroll
                                for (int c = 0; c < 3; c++) xj[c] = operand((unsigned)(3 * j + c));
                            });
                        x = operand(e);
                    }
                    // the entry's result (the diagonal block is the identity) and its dot products
                    if (act && !wait_failed) {
                        if (mode == kSweepInit) {
                            const VT r = x - (x + y);   // r = b - M^-1 A u with u = b
                            KI.vec[4][e] = r;
                            q[e] = r;
                            KI.vec[6][e] = r;
                            v0 += (double)r * (double)r;
                            v1 = max_abs(v1, (double)r);
                            v2 = max_abs(v2, (double)x);
                        } else {
                            const VT w = x + y;
                            if (mode == kSweepS) {
                                As[e] = w;
                                v0 += (double)w * (double)x;
                                v1 += (double)w * (double)w;
                                v2 += (double)w * (double)qe;
                            } else {
                                KI.vec[mode == kSweepUpdate ? 9 - cur : 8 + cur][e] = w;
                                v0 += (double)qe * (double)w;
                            }
                        }
                    }
                }
            }
            seen += (unsigned)nt;
            // virtual CTA v's sums of the sweep, published (the next fill has a barrier)
            {
                const bool max1 = mode != kSweepS, max2 = mode == kSweepInit;
                warp_combine3(v0, v1, v2, max1, max2);
                if (lane == 0) {
                    red[warp] = v0;
                    red[kKrylovWarps + warp] = v1;
                    red[2 * kKrylovWarps + warp] = v2;
                }
                // the pause request: after this iteration's first reduction (which every CTA reaches
                // after its last look at it) and before its second one (which every CTA passes before
                // its next look)
                if (mode == kSweepS && src.done_counter() && pl == 0 && tid == 0 && *(volatile int*)&ctl->pause_at == 0 &&
                    *(volatile unsigned*)src.done_counter() >= src.pause_threshold())
                    *(volatile int*)&ctl->pause_at = C.it;
                bar_rows();   // every warp's sums, and its stores of the sweep's vectors
                if (warp == 0) {
                    // zeros fill the tree (sums, or maxima of absolute values)
                    v0 = lane < kKrylovWarps ? red[lane] : 0.0;
                    v1 = lane < kKrylovWarps ? red[kKrylovWarps + lane] : 0.0;
                    v2 = lane < kKrylovWarps ? red[2 * kKrylovWarps + lane] : 0.0;
                    warp_combine3(v0, v1, v2, max1, max2);
                    if (lane < 3) {
                        asm volatile("fence.acq_rel.gpu;" ::: "memory");
                        const unsigned tag = (C.nred + 1u) | (*(volatile int*)&s_go ? kTagError : 0u);
                        publish(K.part + ((size_t)(C.nred & 1u) * VG + v) * 8 + 2 * lane, lane == 0 ? v0 : lane == 1 ? v1 : v2, tag);
                    }
                }
                v0 = v1 = v2 = 0.0;
            }
        }
        // Every virtual CTA's sums, one slot per thread of the first warps; the control warp combines
        // them and takes the solve's decisions, the same in every CTA of the instance; the barrier
        // hands them to the other warps.
        const int pollers = min((VG + 31) / 32, kKrylovWarps);
        if (warp < pollers) {
            const bool max1 = mode != kSweepS, max2 = mode == kSweepInit;
            double s0 = 0.0, s1 = 0.0, s2 = 0.0;   // lanes past the last slot: sums, or maxima of absolute values
            bool err = false;
            const unsigned n = C.nred + 1u;
            long long spins = 0;
#pragma unroll 1
            for (int j = tid; j < VG && !err; j += 32 * pollers) {
                const double* slot = K.part + ((size_t)(C.nred & 1u) * VG + j) * 8;
                double t0, t1, t2;
#pragma unroll 1
                for (;;) {
                    bool e1, e2;
                    const bool b0 = peek(slot, n, t0, err), b1 = peek(slot + 2, n, t1, e1), b2 = peek(slot + 4, n, t2, e2);
                    if (b0 && b1 && b2) break;
                    if (++spins >= bar_limit || ((spins & 63) == 0 && *(volatile int*)&ctl->err)) {
                        atomicExch(&ctl->err, 1);
                        err = true;
                        t0 = t1 = t2 = 0.0;
                        break;
                    }
                }
                s0 += t0;
                s1 = max1 ? (t1 > s1 ? t1 : s1) : s1 + t1;
                s2 = max2 ? (t2 > s2 ? t2 : s2) : s2 + t2;
            }
            err = __any_sync(0xffffffffu, err);
            warp_combine3(s0, s1, s2, max1, max2);
            if (pollers > 1) {
                if (lane == 0) {
                    s_poll[warp] = s0;
                    s_poll[kKrylovWarps + warp] = s1;
                    s_poll[2 * kKrylovWarps + warp] = s2;
                    if (err) s_poll[3 * kKrylovWarps + warp] = 1.0;
                    else s_poll[3 * kKrylovWarps + warp] = 0.0;
                }
                bar_sync_n(kBarPoll, 32 * pollers);
                if (warp == 0)
#pragma unroll 1
                    for (int j = 1; j < pollers; j++) {
                        const double t0 = s_poll[j], t1 = s_poll[kKrylovWarps + j], t2 = s_poll[2 * kKrylovWarps + j];
                        s0 += t0;
                        s1 = max1 ? (t1 > s1 ? t1 : s1) : s1 + t1;
                        s2 = max2 ? (t2 > s2 ? t2 : s2) : s2 + t2;
                        err |= s_poll[3 * kKrylovWarps + j] != 0.0;
                    }
            }
            if (warp == 0) {
                int next = kSweepS;
                if (err) {
                    next = kSweepFail;
                } else if (mode == kSweepS) {
                    const double omega = s0 / s1;
                    const double rho = -1.0 * omega * s2;
                    const double beta = (rho * C.alpha) / (C.rho * omega);
                    next = kSweepUpdate;
                    __syncwarp();
                    if (lane == 0) {
                        C.omega = omega;
                        C.rho = rho;
                        C.beta = beta;
                    }
                } else {
                    // the stopping test of the start and of an updated residual.  best: the best iterate
                    // so far -- past its attainable accuracy BiCGSTAB's residual drifts back up, so on
                    // stagnation (no new best for kStall iterations) or at max_lin_it the best one is used.
                    // It is kept by leaving it where it is: when an iteration sets a new best (`pending`), the
                    // next update writes the iterate it makes to the other copy of u.
                    const int it = C.it;
                    double rho = C.rho;
                    bool go = true;
                    if (mode != kSweepPlain) {
                        const double rnorm = s1;
                        const double tol = mode == kSweepInit ? K.atol + s2 * rtol : C.tol;
                        const bool better = mode == kSweepInit || rnorm < C.best;
                        const int best_it = mode == kSweepInit ? 0 : better ? it : C.best_it;
                        go = rnorm > tol && it < K.maxit && it - best_it < kStall;
                        __syncwarp();
                        if (lane == 0) {
                            C.rnorm = rnorm;
                            C.tol = tol;
                            if (mode == kSweepUpdate) C.ucur ^= C.pending;   // where the sweep put the iterate
                            C.pending = better;
                            C.best_it = best_it;
                            if (better) C.best = rnorm;
                            if (mode == kSweepInit) {
                                C.rho = s0;
                                if (pl == 0) ctl->bnorm = s2;   // read back with the outcome
                            } else {
                                C.cur = cur ^ 1;
                            }
                        }
                        if (mode == kSweepInit) next = kSweepPlain;
                    }
                    if (!go) next = kSweepEnd;
                    else if (mode != kSweepInit && lane == 0) {
                        C.it = it + 1;
                        C.alpha = rho / s0;
                    }
                }
                // a pause requested before the last iteration's second reduction, at an iteration's top
                if (src.done_counter() && (next == kSweepUpdate || next == kSweepPlain)) {
                    int at = 0;
                    if (lane == 0) at = *(volatile int*)&ctl->pause_at;
                    at = __shfl_sync(0xffffffffu, at, 0);
                    if (at != 0 && C.it >= at) {
                        if (pl == 0 && lane == 0) {
                            ctl->s_rnorm = C.rnorm;
                            ctl->s_tol = C.tol;
                            ctl->s_rho = C.rho;
                            ctl->s_alpha = C.alpha;
                            ctl->s_omega = C.omega;
                            ctl->s_beta = C.beta;
                            ctl->s_best = C.best;
                            ctl->s_it = C.it;
                            ctl->s_best_it = C.best_it;
                            ctl->s_pending = C.pending;
                            ctl->s_upd = next == kSweepUpdate;
                            ctl->s_cur = C.cur;
                            ctl->s_ucur = C.ucur;
                            ctl->s_nred = (int)(C.nred + 1u);
                            ctl->paused = 1;
                        }
                        next = kSweepPause;
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    C.nred++;
                    C.next = next;
                    if (next >= kSweepEnd) *(volatile int*)&s_stop = 1;   // the copy warp may go
                }
            }
        }
        bar_rows();
    }
    if (C.next != kSweepEnd) return;   // paused, or a wait ran out
    const double rnorm = C.rnorm, tol = C.tol;
    const int it = C.it;
    const bool pending = C.pending != 0;
    const double best = C.best;
    const bool conv = rnorm <= tol;
    // x = S u; state += x; sol = -x.  Without convergence the best iterate is u itself when
    // the last iteration set it, else the other copy.
    const VT* ux = KI.vec[C.ucur ^ (conv || pending ? 0 : 1)];
#pragma unroll 1
    for (int r = pl * kKrylovRowThreads + tid; r < V; r += np * kKrylovRowThreads) {
        const int i = K.order ? __ldg(K.order + r) : r;
        const double x0 = (double)ldv(ux + 3 * r) * K.S[3 * i];
        const double x1 = (double)ldv(ux + 3 * r + 1) * K.S[3 * i + 1];
        const double x2 = (double)ldv(ux + 3 * r + 2) * K.S[3 * i + 2];
        if (K.apply_inc) {
            K.u[i] += x0;
            K.v[i] += x1;
            K.h[i] += x2;
            K.sol[3 * i] = -x0;
            K.sol[3 * i + 1] = -x1;
            K.sol[3 * i + 2] = -x2;
        } else {
            K.sol[3 * i] = x0;
            K.sol[3 * i + 1] = x1;
            K.sol[3 * i + 2] = x2;
        }
    }
    if (pl == 0 && tid == 0) {
        ctl->iterations = it;
        ctl->converged = conv ? 1 : 0;
        ctl->rnorm = conv ? rnorm : best;
    }
    if (src.done_counter() && tid == 0) atomicAdd(src.done_counter(), 1u);   // this CTA's instance is done
}

}  // namespace sw2
