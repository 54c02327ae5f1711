// ccz4_tma_tiles0.cu -- the TMA stage kernel (ccz4_stage_tma.cuh) on tile set 0
// (ccz4_kernels.h): 16-wide tiles; also the store epilogue.
// Three ring slots per mixed warpgroup leave the per-point body's local memory
// an L1 of over 70 KB; the FP64 kernels have two warpgroups and take four
// (478 us with three, 470 with four on 128 x 128 x 64 points).
#include "ccz4_stage_tma.cuh"

namespace granite_b200 {
using Ops0 = TmaKernelOps<TmaKernelT<3, TMA_SLOTS_MIXED, false>, TmaKernelT<2, TMA_SLOTS_FP64, false>>;
cudaError_t configure_tma_tiles0(int nsm, TmaGrids& grids) { return Ops0::configure<true>(nsm, grids); }
cudaError_t launch_tma_tiles0(int pm, int epi, bool sel, const DevBlock* blocks, const Tile* tiles, int ntiles,
                              const StageArgs& args, cudaStream_t stream, int grid) {
    return Ops0::launch<true>(pm, epi, sel, blocks, tiles, ntiles, args, stream, grid);
}
}  // namespace granite_b200
