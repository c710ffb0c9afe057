// sw2_halo.h -- how a Krylov solve's rows are shared out, and what each share reads (host code, no
// CUDA).
//
// The node rows come in tiles of kHaloTileRows.  Virtual CTA v of `vgrid` owns the consecutive
// tiles [halo_tile0(v), halo_tile0(v + 1)), cut into `nsub` sub-ranges of which one at a time has
// its operand in shared memory: the vector the sweep multiplies, at the sub-range's own rows and
// at its halo, the other rows its blocks refer to.  Consecutive rows of a mesh numbered with any
// locality refer mostly to each other, so a sweep reads a row's operand from L2 about once instead
// of once per neighbour.  lcol numbers each off-diagonal block's column in that buffer: row r0 + l
// is l, halo row h is (own rows) + h.
#pragma once
#include <algorithm>
#include <vector>

namespace sw2 {

constexpr int kHaloTileRows = 32;
// first of nt tiles that part p of `parts` owns
inline int halo_tile0(int p, int parts, int nt) { return (int)((long long)p * nt / parts); }

struct HaloTables {
    int nsub = 0;                       // sub-ranges per virtual CTA; 0: no sub-division fits
    int max_rows = 0;                   // largest buffer, in rows (own and halo)
    std::vector<int> ptr, idx;          // halo rows of sub-range v * nsub + s, ascending
    std::vector<unsigned short> lcol;   // per off-diagonal block
};

// The tables of an off-diagonal pattern (rp, col; V rows) for `vgrid` virtual CTAs, with the fewest
// sub-ranges whose buffers hold at most cap_rows rows (nsub = 0 when even single tiles need more).
inline void build_halo(int V, const int* rp, const int* col, int vgrid, int cap_rows, HaloTables& t) {
    t = HaloTables();
    const int nt = (V + kHaloTileRows - 1) / kHaloTileRows;
    const int most = (nt + vgrid - 1) / vgrid;   // tiles of the largest virtual CTA
    std::vector<int> mark(V, -1), at(V);
    int stamp = 0;
    // steps of a quarter, the last attempt the division into single tiles
    for (int nsub = std::min(most, std::max(1, (most * kHaloTileRows + cap_rows - 1) / cap_rows));; nsub = std::min(most, nsub + std::max(1, nsub / 4))) {
        t.ptr.assign(1, 0);
        t.idx.clear();
        t.lcol.assign(rp[V], 0);
        t.max_rows = 0;
        bool fits = true;
        for (int v = 0; v < vgrid && fits; v++) {
            const int a = halo_tile0(v, vgrid, nt), b = halo_tile0(v + 1, vgrid, nt);
            for (int s = 0; s < nsub && fits; s++, stamp++) {
                const int r0 = std::min(V, (a + halo_tile0(s, nsub, b - a)) * kHaloTileRows);
                const int r1 = std::min(V, (a + halo_tile0(s + 1, nsub, b - a)) * kHaloTileRows);
                const size_t h0 = t.idx.size();
                for (int k = rp[r0]; k < rp[r1]; k++) {
                    const int j = col[k];
                    if (j >= r0 && j < r1) t.lcol[k] = (unsigned short)(j - r0);
                    else if (mark[j] != stamp) {
                        mark[j] = stamp;
                        t.idx.push_back(j);
                    }
                }
                std::sort(t.idx.begin() + h0, t.idx.end());
                const int rows = r1 - r0 + (int)(t.idx.size() - h0);
                fits = rows <= cap_rows;
                t.max_rows = std::max(t.max_rows, rows);
                for (size_t h = h0; h < t.idx.size(); h++) at[t.idx[h]] = r1 - r0 + (int)(h - h0);
                for (int k = rp[r0]; fits && k < rp[r1]; k++)
                    if (col[k] < r0 || col[k] >= r1) t.lcol[k] = (unsigned short)at[col[k]];
                t.ptr.push_back((int)t.idx.size());
            }
        }
        if (fits) {
            t.nsub = nsub;
            return;
        }
        if (nsub >= most) break;
    }
    t = HaloTables();
}

}  // namespace sw2
