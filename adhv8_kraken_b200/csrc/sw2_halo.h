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
#include <cmath>
#include <cstdint>
#include <utility>
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

// the nodes along the Morton curve of their coordinates: order[new] = old
inline std::vector<int> morton_order(int V, const double* x, const double* y) {
    auto spread = [](uint64_t v) {   // a zero between any two of the low 32 bits
        v = (v | v << 16) & 0x0000ffff0000ffffull;
        v = (v | v << 8) & 0x00ff00ff00ff00ffull;
        v = (v | v << 4) & 0x0f0f0f0f0f0f0f0full;
        v = (v | v << 2) & 0x3333333333333333ull;
        return (v | v << 1) & 0x5555555555555555ull;
    };
    const auto bx = std::minmax_element(x, x + V), by = std::minmax_element(y, y + V);
    const double x0 = *bx.first, y0 = *by.first, span = std::max(std::max(*bx.second - x0, *by.second - y0), 1e-300);
    std::vector<std::pair<uint64_t, int>> key(V);
    for (int i = 0; i < V; i++) {
        const double fx = (x[i] - x0) / span * 4294967295.0, fy = (y[i] - y0) / span * 4294967295.0;
        key[i] = {spread((uint64_t)fx) | spread((uint64_t)fy) << 1, i};
    }
    std::sort(key.begin(), key.end());
    std::vector<int> order(V);
    for (int i = 0; i < V; i++) order[i] = key[i].second;
    return order;
}

// The share tables of a mesh.  A numbering without locality has more halo rows than own ones, and every
// sweep reads each of them from L2 (up to four vectors' entries): the solve then takes the rows in
// Morton order of their nodes, if that halves the halos (16k nodes row by row, 1.6 halo rows per own
// one: 17.9 -> 17.0 us per iteration; 500k 203 -> 141).  Small shares have as many halo rows in any
// order, and up to five tiles' worth are fetched at once: left alone (a channel of 2,600 nodes, 1.5
// halo rows per own one, 96 per virtual CTA: 1 % slower reordered).
// order[new] = old where the order is not the nodes' own, else empty; rp, col become the pattern in the
// order used (blocks of a row stay in the order they had).
constexpr int kHaloFew = 5 * kHaloTileRows;
inline void build_shares(int V, std::vector<int>& rp, std::vector<int>& col, const double* x, const double* y, int vgrid,
                         int cap_rows, HaloTables& t, std::vector<int>& order) {
    order.clear();
    build_halo(V, rp.data(), col.data(), vgrid, cap_rows, t);
    if (t.nsub > 0 && t.idx.size() <= std::max((size_t)V, (size_t)kHaloFew * vgrid)) return;
    std::vector<int> ord = morton_order(V, x, y), at(V), prp(1, 0), pcol;
    for (int i = 0; i < V; i++) at[ord[i]] = i;
    prp.reserve(V + 1);
    pcol.reserve(col.size());
    for (int i = 0; i < V; i++) {
        for (int k = rp[ord[i]]; k < rp[ord[i] + 1]; k++) pcol.push_back(at[col[k]]);
        prp.push_back((int)pcol.size());
    }
    HaloTables p;
    build_halo(V, prp.data(), pcol.data(), vgrid, cap_rows, p);
    if (p.nsub == 0 || (t.nsub > 0 && 2 * p.idx.size() > t.idx.size())) return;
    t = std::move(p);
    rp.swap(prp);
    col.swap(pcol);
    order.swap(ord);
}

}  // namespace sw2
