// ccz4_tma_grids.h -- which kernels of a TMA tile set may be launched on a device.
#pragma once

namespace granite_b200 {

// The persistent grid of every kernel of a tile set, by precision mode, epilogue,
// per-tile precision and whether the stencil coefficients come from the kernel
// arguments; 0 = not to be launched. Each kernel has its own entry: the register
// split of one build says nothing about its twin's, and a kernel whose split does
// not add up would wait for registers that never free up.
struct TmaGrids {
    int grid[3][2][2][2];
    bool refused;  // a kernel of the set may not be launched
    void put(int pm, int epi, bool sel, bool uniform, int registers, int needed, int g) {
        const bool ok = registers == needed;
        grid[pm][epi][sel][uniform] = ok ? g : 0;
        if (!ok) refused = true;
    }
    int of(int pm, int epi, bool sel, bool uniform) const { return grid[pm][epi][sel][uniform]; }
};

}  // namespace granite_b200
