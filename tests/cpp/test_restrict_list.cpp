// The list of restricted cells (ccz4_restrict_list.h): the cells and sources that
// the boxes leave when they are applied one after the other, in block order, and
// no more memory on the way than the list and one block's table.
#include <array>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <new>
#include <random>
#include <utility>

#include "ccz4_restrict_list.h"

static size_t held = 0, peak = 0;
void* operator new(size_t n) {
    size_t* p = static_cast<size_t*>(std::malloc(n + 16));
    if (!p) throw std::bad_alloc();
    *p = n;
    held += n;
    peak = held > peak ? held : peak;
    return reinterpret_cast<char*>(p) + 16;
}
void operator delete(void* q) noexcept {
    if (!q) return;
    size_t* p = reinterpret_cast<size_t*>(static_cast<char*>(q) - 16);
    held -= *p;
    std::free(p);
}
void operator delete(void* q, size_t) noexcept { operator delete(q); }

using namespace granite_b200;

int main() {
    constexpr int BLOCKS = 60, FINE = 60;
    std::mt19937 rng(7);
    auto pick = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
    std::vector<std::array<int, 3>> total(BLOCKS + FINE);
    for (auto& t : total)
        for (int d = 0; d < 3; ++d) t[d] = pick(24, 36);
    auto cells = [&](int b, int d) { return total[(size_t)b][(size_t)d]; };
    std::vector<XferBox> boxes;  // fine block by fine block, each over a few coarse blocks; they overlap
    for (int f = 0; f < FINE; ++f)
        for (int q = 0; q < 3; ++q) {
            XferBox x{};
            x.src = BLOCKS + f;
            x.dst = pick(0, BLOCKS - 1);
            for (int d = 0; d < 3; ++d) {
                x.n[d] = pick(0, 9);
                x.d0[d] = pick(0, cells(x.dst, d) - x.n[d]);
                x.s0[d] = pick(0, cells(x.src, d) - 2 * x.n[d]);
            }
            boxes.push_back(x);
        }
    size_t volume = 0, table = 0;
    for (const auto& x : boxes) volume += (size_t)x.n[0] * x.n[1] * x.n[2];
    for (int b = 0; b < BLOCKS; ++b) table = std::max(table, (size_t)cells(b, 0) * cells(b, 1) * cells(b, 2));

    const size_t before = held;
    peak = held;
    const std::vector<GhostSrc> list = restriction_list(boxes, cells);
    // the list, one table (and its predecessor while it grows), the boxes' order
    const size_t most = (volume + 2 * table) * sizeof(GhostSrc) + boxes.size() * 64;
    int bad = peak - before > most;
    if (bad) std::printf("peak %zu bytes, at most %zu\n", peak - before, most);

    std::map<std::pair<int, int>, std::pair<int, int>> want;
    for (const auto& x : boxes)
        for (int k = 0; k < x.n[2]; ++k)
            for (int j = 0; j < x.n[1]; ++j)
                for (int i = 0; i < x.n[0]; ++i) {
                    const int dc = x.d0[0] + i + cells(x.dst, 0) * (x.d0[1] + j + cells(x.dst, 1) * (x.d0[2] + k));
                    const int sc = x.s0[0] + 2 * i + cells(x.src, 0) * (x.s0[1] + 2 * j + cells(x.src, 1) * (x.s0[2] + 2 * k));
                    want[{x.dst, dc}] = {x.src, sc};
                }
    bad += want.size() != list.size() || want.size() == volume;  // (some boxes do overlap)
    auto it = want.begin();
    for (size_t q = 0; q < list.size() && it != want.end(); ++q, ++it)
        bad += it->first != std::make_pair(list[q].dst_block, list[q].dst_cell) ||
               it->second != std::make_pair(list[q].src_block, list[q].src_cell);
    bad += !restriction_list(std::vector<XferBox>{}, cells).empty();
    std::printf(bad ? "%d wrong\n" : "OK\n", bad);
    return bad != 0;
}
