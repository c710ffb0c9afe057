// sw2_layout.h -- how a Krylov launch lays out its shared memory (host code, no CUDA).
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

namespace sw2 {

// the tile records a warp group's ring holds at each of its places, and the operand buffer
struct RingLayout {
    int stages = 0;                          // 0: sweeps from global memory
    unsigned stage_bytes = 0, x_bytes = 0;   // one tile record, the operand buffer
    size_t smem = 0;
};
// what an instance asks of the staged sweeps; one solved without them (banded, D-ILU) asks nothing
struct RingNeed {
    bool krylov;
    unsigned record_bytes;   // its largest tile record
    unsigned x_bytes;        // its largest operand buffer
    bool fits;               // its shares could be cut to the buffer's cap (sw2_halo.h)
};

// The layout for the instances of a runner: `want` places and one (-1: the deepest ring that fits
// `limit` bytes) for each of `groups` warp groups, falling back to the shallower ring and to none.
// It stays at least as large as `last`, a layout in use before: instances come and go.
inline RingLayout ring_layout(const std::vector<RingNeed>& needs, int want, int groups, size_t limit, const RingLayout& last) {
    RingLayout r;
    unsigned record = 16, x = 0;
    bool fits = true;
    for (const RingNeed& n : needs) {
        if (!n.krylov) continue;
        record = std::max(record, n.record_bytes);
        x = std::max(x, n.x_bytes);
        fits = fits && n.fits;
    }
    if (!fits || want == 0) return r;
    r.stage_bytes = std::max((record + 127u) & ~127u, last.stage_bytes);
    r.x_bytes = std::max(x, last.x_bytes);
    auto bytes = [&](int stages) { return (size_t)(stages - 1) * groups * r.stage_bytes + r.x_bytes; };
    r.stages = want < 0 ? 3 : want;   // the deepest: a CTA whose tiles all stay in its ring copies them once
    if (bytes(r.stages) > limit) r.stages = 2;
    if (bytes(r.stages) > limit) return last.stages ? ring_layout(needs, want, groups, limit, RingLayout()) : RingLayout();
    r.smem = bytes(r.stages);
    return r;
}

}  // namespace sw2
