// Every kernel of a tile set answers for itself (ccz4_tma_grids.h): one built with
// other registers than its split needs is not launched, whatever its twins are.
#include <cstdio>

#include "ccz4_tma_grids.h"

int main() {
    int bad = 0;
    for (int off = 0; off < 24; ++off) {  // the kernel whose register count is off
        granite_b200::TmaGrids g{};
        int k = 0;
        // in the order in which the kernels are configured: coefficients from the descriptors first
        for (int uniform = 0; uniform < 2; ++uniform)
            for (int pm = 0; pm < 3; ++pm)
                for (int epi = 0; epi < 2; ++epi)
                    for (int sel = 0; sel < 2; ++sel, ++k) g.put(pm, epi, sel, uniform, k == off ? 160 : 168, 168, 148);
        k = 0;
        for (int uniform = 0; uniform < 2; ++uniform)
            for (int pm = 0; pm < 3; ++pm)
                for (int epi = 0; epi < 2; ++epi)
                    for (int sel = 0; sel < 2; ++sel, ++k) bad += g.of(pm, epi, sel, uniform) != (k == off ? 0 : 148);
        bad += !g.refused;
    }
    granite_b200::TmaGrids all{};
    all.put(0, 1, false, true, 168, 168, 148);
    bad += all.refused || all.of(0, 1, false, true) != 148 || all.of(0, 1, false, false) != 0;
    std::printf(bad ? "%d wrong\n" : "OK\n", bad);
    return bad != 0;
}
