// knc_runs.h — the row-walking recovery's work list (host).
#pragma once

#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

#include "knc_internal.h"

namespace knc {

struct RecoveryRuns {
    std::vector<int4> runs;   // {slot, i0, j0, rows} of 32 columns
    std::vector<int> off;     // warp k walks runs off[k] .. off[k + 1] - 1; a whole number of CTAs of warps
};

// The blocks' columns of 32 zones, one after the other, cut into as many equal
// runs of whole rows as the device holds warps of the recovery (`ctas` CTAs; a
// column's end cuts too). A run's first rows wait for memory with nothing to
// compute, so a warp has one or two, not one per tile, and all warps end
// together. Where a block's columns fill CTAs, the warps of a CTA walk the same
// rows of neighbouring columns; the other blocks' columns follow in CTAs of
// their own, and the runs get longer until both fit (no second wave). Against
// 8-row tiles strided over the same warps (4.5 tiles a warp on the 4096 x 1024
// wind, 1.1 on the 2048 x 512 jet): folds of 20 wind steps 9.93 -> 9.87 ms on the
// device (9.98 with every column on its own), 10 jet steps 3.68 -> 3.53, 2 RK3
// steps of uneven blocks 1.33 -> 1.28.
inline RecoveryRuns recovery_runs(const std::vector<std::pair<int64_t, int64_t>>& shapes, int64_t ctas) {
    constexpr int WPC = TILE_THREADS / 32;
    auto columns = [](int64_t nq) { return (nq + TILE_Q - 1) / TILE_Q; };
    // rows to walk: by `WPC` neighbouring warps at once, by single warps
    int64_t wide = 0, single = 0;
    for (const auto& s : shapes) {
        const int64_t cols = columns(s.second);
        if (cols % WPC == 0) wide += s.first * (cols / WPC);
        else single += s.first * cols;
    }
    auto groups = [](int64_t rows, int64_t per) { return (rows + per - 1) / per; };
    auto ctas_of = [&](int64_t per) { return groups(wide, per) + (groups(single, per) + WPC - 1) / WPC; };
    int64_t per = std::max<int64_t>(1, groups(WPC * wide + single, ctas * WPC));
    while (ctas_of(per) > std::max<int64_t>(ctas, 2)) ++per;
    RecoveryRuns out;
    std::vector<int4> pieces;
    std::vector<size_t> first;   // of a group's pieces
    out.off.reserve((size_t)(ctas_of(per) * WPC + 1));
    for (int width : {WPC, 1}) {
        pieces.clear();
        first.clear();
        int64_t done = 0;   // rows given to each of `width` neighbouring warps
        for (size_t k = 0; k < shapes.size(); ++k) {
            const int64_t nr = shapes[k].first, nq = shapes[k].second;
            if ((columns(nq) % WPC == 0 ? WPC : 1) != width) continue;
            for (int64_t j0 = 0; j0 < nq; j0 += width * TILE_Q)
                for (int64_t i0 = 0; i0 < nr;) {
                    if (done % per == 0) first.push_back(pieces.size());
                    const int64_t rows = std::min(nr - i0, per - done % per);
                    pieces.push_back(make_int4((int)k, (int)i0, (int)j0, (int)rows));
                    i0 += rows;
                    done += rows;
                }
        }
        first.push_back(pieces.size());
        out.runs.reserve(out.runs.size() + pieces.size() * width);
        for (size_t g = 0; g + 1 < first.size(); ++g)
            for (int w = 0; w < width; ++w) {
                out.off.push_back((int)out.runs.size());
                for (size_t p = first[g]; p < first[g + 1]; ++p) {
                    int4 r = pieces[p];
                    r.z += w * TILE_Q;
                    out.runs.push_back(r);
                }
            }
        while (out.off.size() % WPC) out.off.push_back((int)out.runs.size());   // whole CTAs
    }
    out.off.push_back((int)out.runs.size());
    return out;
}

}  // namespace knc
