// ccz4_restrict_list.h -- the list of a level's restricted cells. Host code only.
#pragma once

#include <algorithm>
#include <numeric>
#include <vector>

#include "ccz4_kernels.h"

namespace granite_b200 {

// The restriction boxes into a level (x.dst coarse, x.src fine, children of the
// box's first cell at x.s0) as one list with each coarse cell once, block after
// block: where boxes overlap the last one decides, as when they run one after the
// other (a box reads only cells of the finer level). cells(b, d): block b's cells
// along axis d, ghosts included. Besides the list it holds one coarse block's table.
template <typename Cells>
std::vector<GhostSrc> restriction_list(const std::vector<XferBox>& boxes, const Cells& cells) {
    std::vector<int> order(boxes.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return boxes[a].dst < boxes[b].dst; });
    size_t most = 0;  // the list's length, or more where boxes overlap
    for (const XferBox& x : boxes) most += (size_t)x.n[0] * x.n[1] * x.n[2];
    std::vector<GhostSrc> items;
    items.reserve(most);
    std::vector<GhostSrc> table;  // of the coarse block at hand
    for (size_t at = 0; at < order.size();) {
        const int dst = boxes[order[at]].dst;
        const int T0 = cells(dst, 0), T1 = cells(dst, 1), T2 = cells(dst, 2);
        table.assign((size_t)T0 * T1 * T2, GhostSrc{-1, 0, 0, 0});
        for (; at < order.size() && boxes[order[at]].dst == dst; ++at) {
            const XferBox& x = boxes[order[at]];
            const int S0 = cells(x.src, 0), S1 = cells(x.src, 1);
            for (int k = 0; k < x.n[2]; ++k)
                for (int j = 0; j < x.n[1]; ++j)
                    for (int i = 0; i < x.n[0]; ++i) {
                        const int cell = x.d0[0] + i + T0 * (x.d0[1] + j + T1 * (x.d0[2] + k));
                        table[cell] = GhostSrc{dst, cell, x.src,
                                               x.s0[0] + 2 * i + S0 * (x.s0[1] + 2 * j + S1 * (x.s0[2] + 2 * k))};
                    }
        }
        for (const GhostSrc& g : table)
            if (g.dst_block >= 0) items.push_back(g);
    }
    return items;
}

}  // namespace granite_b200
