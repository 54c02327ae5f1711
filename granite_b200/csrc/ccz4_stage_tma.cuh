// ccz4_stage_tma.cuh -- the TMA stage kernel.
//
// One CTA per SM: NWG compute warpgroups (128 threads, one 16 x 4 x 2 tile
// each) and one warpgroup of load warps, load warp g serving compute
// warpgroup g. Each pair is independent of the others: it walks its own tiles
// (CTA b's warpgroup g: list entries g gridDim.x + b, + gridDim.x NWG, ...) through
// its own ring of field boxes.
//
//   load warp:   finds the next tile (with per-tile precision the next one whose
//                flag the launch takes, a ballot over 32 flags at a time),
//                copies it and its block's descriptor into shared memory one round
//                ahead, and per field waits until the slot is empty and issues
//                the field's three box loads (TileBoxes);
//   compute warps: per field wait for the slot's boxes, evaluate the stencils,
//                arrive on the slot's empty barrier (one arrival per warp) and
//                go on; no barrier among the warps. The algebra is ccz4_point.
//
// What bounds it: instruction issue (67 % of the slots) and latency at 12 compute
// warps per SM in the mixed form, latency at 8 in the FP64 form. What measured
// (128 x 128 x 64 points, stage 1-3 average, mixed / FP64): 508 / 685 us when two
// CTAs of 128 threads (one of 256) issued their own loads, one 24 x 12 x (tz + 8)
// box per field behind a CTA barrier, with generic loads of the ring and the
// stencil coefficients in global memory; 424 / 523 with shared-space loads,
// coefficients in the kernel arguments and tiles and descriptors copied ahead;
// 343 / 470 with the load warps, three boxes per field, rolled field loops and
// 32-bit shared addresses. Per field a barrier cost a fifth of the stall cycles
// (a third with three boxes to issue). Prefetching the next tile's fields into
// L2 from the load warps: 20 % slower (the burst delays the ring's own loads).
// Ring slots per mixed warpgroup 3 / 4 / 5: 343 / 351 / 375 (they take L1 from the
// per-point body's local memory).
//
// Registers: the launch gives every thread 65536 / threads; setmaxnreg moves
// the load warpgroup's to the compute warpgroups (the shares below add up to at
// most the launch's total, which TmaKernelOps checks).
//
// Every wait is bounded (TMA_WAIT_NS): a thread whose wait gives up records it
// in StageArgs::errflag and skips its later waits; a compute warp then leaves
// at its next tile, and the load warp stops issuing, waits (bounded) for the
// copies it issued and leaves, so the kernel always ends and no copy into shared
// memory outlives the CTA.
#pragma once

#include <cstdint>
#include <type_traits>

#include "ccz4_point.cuh"
#include "ccz4_tma_grids.h"

namespace granite_b200 {

namespace {

// The boxes of one field of a tile of depth TZ in a ring slot (ccz4_kernels.h):
// the main box, then the far planes below and above it.
template <int TZ>
struct TileBoxes {
    static constexpr int BX = TMA_BOX_X, BY = TMA_BOX_Y;
    static constexpr int MAIN = BX * BY * (TZ + 2), ARM = TMA_ARM_X * TMA_ARM_Y * TMA_ARM_Z;
    static constexpr int CELLS = MAIN + 2 * ARM;
    static_assert(MAIN * sizeof(double) % 128 == 0 && ARM * sizeof(double) % 128 == 0, "boxes stay 128-byte aligned");
    // offset of tile point (x, y, z)
    static __device__ __forceinline__ int point(int x, int y, int z) { return (x + 4) + BX * ((y + 4) + BY * (z + 1)); }
    static __device__ __forceinline__ int plane(int x, int y, int z) {
        const int a = x + TMA_ARM_X * y, p = TMA_ARM_X * TMA_ARM_Y;
        return z < -1 ? MAIN + a + p * (z + 4) : (z > TZ ? MAIN + ARM + a + p * (z - TZ - 1) : point(x, y, z));
    }
    static __device__ __forceinline__ void arms(int x, int y, int z, ArmOffsets& o) {
#pragma unroll
        for (int k = 2; k <= 4; ++k) {
            o.lo[k - 2] = plane(x, y, z - k) * (int)sizeof(double);
            o.hi[k - 2] = plane(x, y, z + k) * (int)sizeof(double);
        }
    }
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// One box of a 4-D tensor map (x, y, z, field) into shared memory.
__device__ __forceinline__ void tma_load_box(unsigned dst, const void* map, int x, int y, int z, int f,
                                             unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(f), "r"(bar)
        : "memory");
}

}  // namespace

}  // namespace granite_b200

#include "ccz4_stage_ring.cuh"

namespace granite_b200 {

namespace {

// NWG compute warpgroups, NBUF ring slots each; REM: x-remainder tiles
// (TMA_REM_X x 4 x 4 points, slots sized for their boxes).
template <int NWG_, int NBUF_, bool REM_>
struct TmaKernelT {
    static constexpr int NWG = NWG_, NBUF = NBUF_;
    static constexpr bool REM = REM_;
    static constexpr int TX = 16, TY = 4, TZ = 2, NP = TX * TY * TZ;
    static constexpr int NTHR = (NWG + 1) * NP;
    static constexpr int BX = TMA_BOX_X, BY = TMA_BOX_Y;
    using Boxes = TileBoxes<TZ>;
    using BoxesRem = TileBoxes<2 * TZ>;
    static_assert(NP == 128 && NWG <= 4 && NBUF <= 4, "one load warp per compute warpgroup");
    static_assert(TMA_REM_X * TY * 2 * TZ == NP, "remainder tiles: one point per thread");
    static constexpr int SLOT = REM ? BoxesRem::CELLS : Boxes::CELLS;
    static constexpr size_t SMEM = (size_t)NWG * NBUF * SLOT * sizeof(double);
    // registers per thread: of the launch, of the load warps, of the compute warps
    static constexpr int LAUNCH_REGS = 65536 / NTHR / 8 * 8;
    static constexpr int LOAD_REGS = 40;  // (24 and 32 spill in the load warps: 8 % slower)
    static constexpr int COMP_REGS = (LAUNCH_REGS * NTHR - LOAD_REGS * NP) / (NWG * NP) / 8 * 8;
    static_assert(NWG * NP * COMP_REGS + NP * LOAD_REGS <= NTHR * LAUNCH_REGS, "the split moves registers, it adds none");
    static_assert(COMP_REGS <= 255 && COMP_REGS >= 128, "compute warps");
};

// The compute warps' stencil source.
template <class C, bool UC>
struct TmaSource {
    static constexpr bool UNROLL = false;
    unsigned slots;  // shared address of the ring's slots
    TmaRing<C::NBUF> ring;
    const StencilCoef& coef;  // UC: the coefficients of every block of the launch, in the kernel arguments
    int lin = 0;
    ArmOffsets arm{};
    int round = 0;

    __device__ __forceinline__ const DevBlock& block() const {
        return *reinterpret_cast<const DevBlock*>(ring.sh.block[round & 1]);
    }
    __device__ __forceinline__ const StencilCoef& coefs() const {
        if constexpr (UC)
            return coef;
        else
            return block();
    }
    template <bool HESS, bool EXACT, bool KOSEP, typename P>
    __device__ __forceinline__ FieldDer<P> der(int /*v*/, const Advection<P, EXACT>& adv) {
        ring.wait();
        const unsigned at = slots + ring.slot * (unsigned)(C::SLOT * sizeof(double));
        const SplitLoad<C::BX, C::BX * C::BY> L{at, at + lin, arm};
        const FieldDer<P> r = field_der_l<P, HESS, true, EXACT, KOSEP>(coefs(), L, adv);
        ring.release();
        return r;
    }
};

}  // namespace

template <int PM, int EPI, class C, bool SEL, bool UC>
__global__ void __launch_bounds__(C::NTHR, 1)
    ccz4_stage_tma_kernel(const DevBlock* __restrict__ blocks, const Tile* __restrict__ tiles, int ntiles,
                         const __grid_constant__ StageArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int g = threadIdx.x / C::NP;  // warpgroup
    if (threadIdx.x < C::NWG) {
        g_tma[threadIdx.x].stop = 0;
        for (int s = 0; s < C::NBUF; ++s) {
            mbar_init(smem_addr(&g_tma[threadIdx.x].full[s]), 1);
            mbar_init(smem_addr(&g_tma[threadIdx.x].empty[s]), C::NP / 32);  // every compute warp arrives
        }
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    __syncthreads();
    const unsigned rings = smem_addr(smem_raw);
    constexpr unsigned RING = C::NBUF * C::SLOT * sizeof(double);
    if (g == C::NWG) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(C::LOAD_REGS));
        const int w = (threadIdx.x - C::NWG * C::NP) / 32;
        if (w < C::NWG) tma_load_warp<C, SEL>(w, blocks, tiles, ntiles, A, rings + w * RING);
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(C::COMP_REGS));
    const int pt = threadIdx.x % C::NP;
    TmaShared& sh = g_tma[g];
    TmaSource<C, UC> S{rings + g * RING, {sh, smem_addr(sh.full), smem_addr(sh.empty), A.errflag}, A.coef};
#pragma unroll 1
    for (int r = 0;; ++r) {
        if (!S.ring.next_round()) break;
        const Tile t = sh.tile[r & 1].t;
        const int ti = sh.tile[r & 1].index;
        if (ti < 0) break;
        S.round = r;
        const DevBlock& B = S.block();
        // this thread's point: 16 x 4 x 2, or TMA_REM_X x 4 x 4 of an x-remainder tile
        int lx, ly, lz;
        if (C::REM && t.w < 0) {
            lx = pt % TMA_REM_X;
            ly = (pt / TMA_REM_X) % C::TY;
            lz = pt / (TMA_REM_X * C::TY);
            C::BoxesRem::arms(lx, ly, lz, S.arm);
        } else {
            lx = pt % C::TX;
            ly = (pt / C::TX) % C::TY;
            lz = pt / (C::TX * C::TY);
            C::Boxes::arms(lx, ly, lz, S.arm);
        }
        S.lin = C::Boxes::point(lx, ly, lz) * (int)sizeof(double);
        const int i = t.i0 + lx, j = t.j0 + ly, k = t.k0 + lz;
        const bool valid = i < B.n[0] && j < B.n[1] && k < B.n[2];
        // pointwise loads of threads outside the block use a valid cell; their results are dropped
        const int ic = min(i, B.n[0] - 1), jc = min(j, B.n[1] - 1), kc = min(k, B.n[2] - 1);
        const long long c = cell_index(B, ic + NG, jc + NG, kc + NG);
        AlgebraT<PM> L[NV];
        point_pm<PM>(B, B.buf[A.in_sel], c, A, S, L);
        const int2 pr = A.push ? A.tile_push[ti] : make_int2(0, 0);
        if (valid) stage_epilogue<EPI>(B, A, c, L, A.push ? A.push + pr.x : nullptr, pr.y, i, j, k);
    }
}

// Launchers of one tile set: C3 the mixed kernels (12 compute warps per SM), C2
// the FP64 ones (8).
template <class C3, class C2>
struct TmaKernelOps {
    template <int PM>
    using Cfg = typename std::conditional<PM == PM_MIXED, C3, C2>::type;
    // the register split needs the launch's full share: setmaxnreg.inc would wait for registers that never free up
    template <int PM, int EPI, bool SEL, bool UC>
    static cudaError_t configure_one(int nsm, TmaGrids& grids) {
        using C = Cfg<PM>;
        auto k = ccz4_stage_tma_kernel<PM, EPI, C, SEL, UC>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e != cudaSuccess) return e;
        cudaFuncAttributes fa{};
        if ((e = cudaFuncGetAttributes(&fa, k))) return e;
        grids.put(PM, EPI, SEL, UC, fa.numRegs, C::LAUNCH_REGS, nsm);
        return cudaSuccess;
    }
    template <int PM, int EPI, bool SEL, bool UC>
    static cudaError_t launch_one(const DevBlock* blocks, const Tile* tiles, int ntiles, const StageArgs& args,
                                  cudaStream_t stream, int grid) {
        using C = Cfg<PM>;
        ccz4_stage_tma_kernel<PM, EPI, C, SEL, UC><<<grid, C::NTHR, C::SMEM, stream>>>(blocks, tiles, ntiles, args);
        return cudaGetLastError();
    }
    template <bool UC>
    static cudaError_t configure_rk(int nsm, TmaGrids& grids) {
        cudaError_t e;
        if ((e = configure_one<PM_FP64, EPI_RK, false, UC>(nsm, grids))) return e;
        if ((e = configure_one<PM_MIXED, EPI_RK, false, UC>(nsm, grids))) return e;
        if ((e = configure_one<PM_MIXED, EPI_RK, true, UC>(nsm, grids))) return e;
        return configure_one<PM_FP64F, EPI_RK, true, UC>(nsm, grids);
    }
    template <bool UC>
    static cudaError_t launch_rk(int pm, bool sel, const DevBlock* blocks, const Tile* tiles, int ntiles,
                                 const StageArgs& args, cudaStream_t stream, int grid) {
        if (pm == PM_FP64 && !sel) return launch_one<PM_FP64, EPI_RK, false, UC>(blocks, tiles, ntiles, args, stream, grid);
        if (pm == PM_MIXED && !sel) return launch_one<PM_MIXED, EPI_RK, false, UC>(blocks, tiles, ntiles, args, stream, grid);
        if (pm == PM_MIXED && sel) return launch_one<PM_MIXED, EPI_RK, true, UC>(blocks, tiles, ntiles, args, stream, grid);
        if (pm == PM_FP64F && sel) return launch_one<PM_FP64F, EPI_RK, true, UC>(blocks, tiles, ntiles, args, stream, grid);
        return cudaErrorInvalidValue;
    }
    // STORE: plus the store epilogue (single-block launches, always uniform).
    template <bool STORE>
    static cudaError_t configure(int nsm, TmaGrids& grids) {
        cudaError_t e;
        if ((e = configure_rk<false>(nsm, grids))) return e;
        if ((e = configure_rk<true>(nsm, grids))) return e;
        if constexpr (STORE) {
            if ((e = configure_one<PM_FP64, EPI_STORE, false, true>(nsm, grids))) return e;
            if ((e = configure_one<PM_MIXED, EPI_STORE, false, true>(nsm, grids))) return e;
        }
        return cudaSuccess;
    }
    template <bool STORE>
    static cudaError_t launch(int pm, int epi, bool sel, const DevBlock* blocks, const Tile* tiles, int ntiles,
                              const StageArgs& args, cudaStream_t stream, int grid) {
        if (epi == EPI_RK) {
            if (args.coef_uniform) return launch_rk<true>(pm, sel, blocks, tiles, ntiles, args, stream, grid);
            return launch_rk<false>(pm, sel, blocks, tiles, ntiles, args, stream, grid);
        }
        if constexpr (STORE) {
            if (!args.coef_uniform || sel) return cudaErrorInvalidValue;
            if (pm == PM_FP64) return launch_one<PM_FP64, EPI_STORE, false, true>(blocks, tiles, ntiles, args, stream, grid);
            if (pm == PM_MIXED) return launch_one<PM_MIXED, EPI_STORE, false, true>(blocks, tiles, ntiles, args, stream, grid);
        }
        return cudaErrorInvalidValue;
    }
};

}  // namespace granite_b200
