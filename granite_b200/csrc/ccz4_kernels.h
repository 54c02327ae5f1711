// ccz4_kernels.h -- host-side launchers of the CCZ4 device kernels.
#pragma once

#include <cuda_runtime.h>

#include "ccz4_common.cuh"

namespace granite_b200 {

enum { EPI_STORE = 0, EPI_RK = 1 };

// Kernel variants of the fused stage: 0 = stencils from global memory
// (32x4x1 tiles), 1 = fields staged through shared memory with cp.async
// (16x4x2 tiles); 2, 3 = variant 0 with the registers capped at 168 / 128 per
// thread (3 / 4 CTAs per SM); 4 = persistent CTAs whose load warps stream every
// field of a 16x4x2 tile and its halo into rings of shared-memory slots with
// TMA (cp.async.bulk.tensor) and mbarriers. The constraint and KO kernels always
// use variant-0 tiles.
enum {
    VARIANT_GLOBAL = 0, VARIANT_SMEM = 1, VARIANT_GLOBAL_R168 = 2, VARIANT_GLOBAL_R128 = 3, VARIANT_TMA = 4,
    NUM_VARIANTS = 5
};

// Tile shape of a stage-kernel variant (points along x, y, z).
void stage_tile_dims(int variant, int* tx, int* ty, int* tz);

// Tile sets of the TMA kernel: 0 = 16 x 4 x 2 tiles (and the store epilogue of the
// drop-in RHS), 1 = with x-remainder tiles: a block whose x extent leaves 8 cells
// after its 16-wide tiles covers them with 8 x 4 x 4 tiles (Tile::w = -8, every
// thread on a point) instead of 16-wide tiles half outside the block.
constexpr int NUM_TMA_TILESETS = 2;
// A configuration id, what a caller may set per precision and block-size class,
// stands for a tile set: those below TMA_FIRST_REM_CFG for set 0, the others for
// set 1. TMA_TILESET_CFG: the id reported for a set that the library chose.
constexpr int NUM_TMA_CFGS = 18, TMA_FIRST_REM_CFG = 11;
constexpr int tma_tileset(int cfg) { return cfg < TMA_FIRST_REM_CFG ? 0 : 1; }
constexpr int TMA_TILESET_CFG[NUM_TMA_TILESETS] = {0, 12};
// Ring slots per compute warpgroup of the mixed and of the FP64 kernels.
constexpr int TMA_SLOTS_MIXED = 3, TMA_SLOTS_FP64 = 4;
constexpr int TMA_TZ = 2;
// Points of an x-remainder tile along x.
constexpr int TMA_REM_X = 8;
// The boxes three tensor-map loads bring in per field of a tile of depth tz:
// 24 x 12 x (tz + 2) cells, the tile with its 4-cell halo in x and y and the one
// plane beyond it on either side in z that the mixed derivatives read off the
// axes; and, below and above it, 16 x 4 x 3, the farther planes, which the z
// stencils read at the tile's own columns only. One 24 x 12 x (tz + 8) box would
// hold 1.6 (tz = 4) or 1.9 (tz = 2) times the cells: as much more shared memory
// per ring slot and L2 traffic per field.
// Tensor maps exist per box shape: shape 0 (tz = 2), shape 1 (tz = 4, the
// remainder tiles) and shape 2, the far planes of every tile.
constexpr int TMA_BOX_X = 16 + 8, TMA_BOX_Y = 4 + 8;
constexpr int TMA_ARM_X = 16, TMA_ARM_Y = 4, TMA_ARM_Z = 3;
constexpr int TMA_SHAPES = 3;
constexpr int TMA_SHAPE_TZ[TMA_SHAPES] = {TMA_TZ, 2 * TMA_TZ, 0};
constexpr int TMA_SHAPE_REM = 1, TMA_SHAPE_ARM = 2;
// Tensor map of one 22-field block buffer (dims x, y, z, field; cells incl.
// ghosts) with box shape `shape`. Returns false when the buffer cannot be
// described (odd x extent, misaligned base) or the block is smaller than a tile
// with its halo; such blocks use the global-load kernel.
bool encode_block_tmap(void* map128, const double* base, const DevBlock& d, int shape);

// Per-device kernel attributes (shared-memory opt-in); call with the device current.
cudaError_t configure_stage_kernels();

// Whether every kernel of the TMA variant may be launched on the current device
// (TmaGrids); without, its blocks use the global-load kernel.
bool tma_available();

// Precision modes of the stage kernels: FP64 algebra with the reference-order
// FP64 stencils, FP32 algebra (mixed), or FP64 algebra with pair-difference
// FP64 stencils (PM_FP64F, RK epilogue only: the FP64 pass of the per-tile
// precision, where parity is with the FP64 path to rounding, not bit for bit).
enum { PM_FP64 = 0, PM_MIXED = 1, PM_FP64F = 2 };

// Fused RHS (+KO) over a tile work-list in precision mode `precision` (PM_*);
// with args.tile_prec set, only the tiles flagged args.want_prec. tileset: the
// TMA tile set (ignored by the other variants); args.tmaps* must hold the tensor
// maps of its box shapes.
cudaError_t launch_stage(int variant, int tileset, int precision, int epi, const DevBlock* blocks,
                         const Tile* tiles, int ntiles, const StageArgs& args, cudaStream_t stream);

// Per-tile precision flags of tiles [first, first + ntiles): flag[ti] = 1 when a
// point of the tile has chi < chi_fp64 in slot `sel` (FP64 algebra), else 0.
cudaError_t launch_classify(int variant, const DevBlock* blocks, const Tile* tiles, int first, int ntiles,
                            int sel, double chi_fp64, unsigned char* flag, cudaStream_t stream);

// KO dissipation only: rhs += KO(u) at interior points of one block.
cudaError_t launch_dissipation(const DevBlock* block, int in_sel, double* rhs, int ntiles,
                               const Tile* tiles, cudaStream_t stream);

// Ghost-cell work items: one per (block, ghost cell); built on the host.
struct GhostItem {
    int block;
    int cell;  // linear cell index within the block (incl. ghosts)
};

enum GhostMode {
    GHOST_ZERO_GRADIENT = 0,    // all faces (amr.cpp:447-480)
    GHOST_SOMMERFELD = 1,       // 1/r falloff (main.cpp:351-463)
    GHOST_PERIODIC = 2,         // periodic wrap (gauge-wave workload)
    GHOST_ZERO_GRADIENT_MASKED = 3  // only the faces flagged in a per-block 6-bit mask
};

// Fill every listed ghost cell of buffer slot `sel` for all 22 fields.
// facemask (per block; bit 2d = low face of axis d, bit 2d+1 = high face) is
// read only by GHOST_ZERO_GRADIENT_MASKED.
cudaError_t launch_ghost_fill(int mode, const DevBlock* blocks, const GhostItem* items, int nitems,
                              int sel, const unsigned char* facemask, cudaStream_t stream);

// A box of cells of block dst filled by trilinear interpolation of block src
// (amr.cpp:484-564). Block-local cell indices including ghosts (s0 is only used
// on the host).
struct XferBox {
    int dst, src;
    int d0[3];
    int s0[3];
    int n[3];
};
// One CTA of a transfer launch: XFER_CHUNK consecutive cells of a box.
struct BoxChunk {
    int box;
    int start;
};
constexpr int XFER_CHUNK = 256;

// Prolongation of slot src_sel of the source blocks into slot dst_sel of the destinations.
cudaError_t launch_prolong(const DevBlock* blocks, const XferBox* boxes, const BoxChunk* chunks, int nchunks, int dst_sel,
                           int src_sel, cudaStream_t stream);

// One ghost cell of a level and where its value comes from (GRANITE_AMR_GHOSTS):
//   src_block >= 0, src_cell >= 0: copy of that cell of a same-level block
//   src_block >= 0, src_cell <  0: prolongation from that coarse block
//   src_block <  0               : the block's own fill (zero-gradient or 1/r falloff)
struct GhostSrc {
    int dst_block, dst_cell, src_block, src_cell;
};

// Every listed ghost cell written once: copies and local fills read slot
// `sel`, prolongations read slot 0 of the coarse block. local_mode:
// GHOST_ZERO_GRADIENT or GHOST_SOMMERFELD. prolong: prolongated cells are
// written in this many slots from sel on (0: not at all).
cudaError_t launch_ghost_sources(const DevBlock* blocks, const GhostSrc* items, long long nitems, int sel,
                                 int local_mode, int prolong, cudaStream_t stream);

// Restriction of slot 0 (amr.cpp:566-626): every listed coarse cell becomes the
// mean of the 2x2x2 fine cells of src_block from src_cell on.
cudaError_t launch_restrict(const DevBlock* blocks, const GhostSrc* items, long long nitems, cudaStream_t stream);

// Constraint monitor (ccz4.cpp:941-1159) over a tile work-list. Writes ham /
// mom (single-block drop-in; may be null) and per-CTA partial sums of H^2 and
// |M|^2 to partials[2 * tile] (may be null).
cudaError_t launch_constraints(const DevBlock* blocks, const Tile* tiles, int ntiles, int sel,
                               double* ham, double* mom, double* partials, cudaStream_t stream);

// Regrid tagger (amr.cpp:653-731) over the interior cells of slot 0 of the
// listed tiles (32x4x1 monitor shape): adds the number of tagged cells to *count.
cudaError_t launch_tag_count(const DevBlock* blocks, const Tile* tiles, int ntiles, int var, double threshold,
                             unsigned long long* count, cudaStream_t stream);

// Matter sources of the CCZ4 RHS from GRMHD primitives (grmhd.cpp:1034-1103)
// at the interior cells of one block. prim: NPRIM fields of B.stride cells.
// Outputs: rho[c], S[c], Si[c * si_cell + a * si_comp], Sij[c * sij_cell + q * sij_comp]
// (the reference's AoS arrays: si_cell 3, si_comp 1, sij_cell 6, sij_comp 1).
constexpr int NPRIM = 11;
struct MatterOut {
    double* rho;
    double* Si;
    double* Sij;
    double* S;
    long long si_cell, si_comp, sij_cell, sij_comp;
};
cudaError_t launch_matter_sources(const DevBlock& B, const double* prim, const MatterOut& out, cudaStream_t stream);

// Psi4Extractor::extract (postprocess.cpp:245-314) on one block: modes[r * nm + q]
// (q over l = 2..l_max, m = -l..l; nm = (l_max + 1)^2 - 4) at the nr radii (device
// array); psi4_scratch holds nr * n_theta * n_phi values; inside_count[r] gets the
// number of sphere points of radius r inside the block. hi: the block's upper corner.
cudaError_t launch_psi4_modes(const DevBlock& B, const double* u, const double hi[3], const double* radii, int nr,
                              int n_theta, int n_phi, int l_max, double2* psi4_scratch, double2* modes,
                              unsigned int* inside_count, cudaStream_t stream);

// Apparent-horizon flow (horizon_finder.cpp:310-449) on one block. tab holds
// sin(theta_i), cos(theta_i) (nth each), sin(phi_j), cos(phi_j) (nph each),
// evaluated by the host's libm.
struct HorizonArgs {
    double center[3];
    double flow_step, rmin;  // 0.05 dx and 1e-6 dx
    double dth, dph;         // pi / nth, 2 pi / nph
    int nth, nph;
};
// iters flow iterations of every surface point from the radii h (updated in
// place): radii after iteration k at hist[k * N + p], max |Theta| of iteration k
// as the bits of a non-negative double in itmax[k] (zeroed here).
cudaError_t launch_horizon_flow(const DevBlock& B, const double* u, const HorizonArgs& a, const double* tab,
                                double* h, int iters, double* hist, unsigned long long* itmax, cudaStream_t stream);
// terms[3 p ..] = area term, J_z term, 1 (0 where chi < 1e-12) of surface point p.
cudaError_t launch_horizon_surface(const DevBlock& B, const double* u, const HorizonArgs& a, const double* tab,
                                   const double* h, double* terms, cudaStream_t stream);
// findAllHorizons' candidate cells (lapse minima below 0.5), up to cap cell indices
// in arbitrary order; *count = all found.
cudaError_t launch_lapse_minima(const DevBlock& B, const double* u, long long* out, unsigned int* count,
                                unsigned int cap, cudaStream_t stream);

// Per field v: out[v] = max |a - b|, out[22 + v] = max |a| over the interior
// cells of slot 0 of blocks a[i], b[i] (i < nblocks, identical geometry), as the
// bits of non-negative doubles; out[44], out[45] = non-finite values in a, in b.
cudaError_t launch_compare_states(const DevBlock* a, const DevBlock* b, int nblocks, unsigned long long* out,
                                  cudaStream_t stream);

// Deterministic fixed-order sum of n partial pairs into out[2].
cudaError_t launch_sum_partials(const double* partials, int n, double* out, cudaStream_t stream);

}  // namespace granite_b200
