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
// after its current tile, and a load warp stops issuing, waits (bounded) for
// the copies it issued and leaves, so the kernel always ends and no copy into
// shared memory outlives the CTA.
#pragma once

#include <cstdint>
#include <type_traits>

#include "ccz4_point.cuh"

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
// Wait limit of one ring slot: 2 s of wall time, then the kernel records the
// failure in StageArgs::errflag and stops waiting (results are then garbage
// and the host reports the error).
constexpr unsigned long long TMA_WAIT_NS = 2000000000ull;
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

__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// Bounded wait for the completion of the phase of parity `parity`; on a timeout
// the failure is recorded. Returns false then. A waiting warp is suspended
// within each attempt (mbarrier.try_wait); the clock is read every 64 of them.
__device__ __forceinline__ bool tma_wait(unsigned bar, unsigned parity, unsigned int* err) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0 = 0;
#pragma unroll 1
    for (unsigned n = 0;; ++n) {
        if (mbar_try_wait(bar, parity)) return true;
        if (n % 64 == 0) {
            const unsigned long long t = global_ns();
            if (n == 0) t0 = t;
            if (t - t0 > TMA_WAIT_NS) {
                if (err) atomicExch(err, 1u);
                return false;
            }
        }
    }
}

// Tile of a compute warpgroup's round r at [r & 1] (index < 0: no more tiles)
// and its block's descriptor.
struct __align__(16) TmaTile {
    Tile t;
    int index;
    int pad[2];
};
constexpr int TMA_MAX_SLOTS = 4;
struct TmaShared {
    unsigned long long full[TMA_MAX_SLOTS], empty[TMA_MAX_SLOTS];
    TmaTile tile[2];
    __align__(16) unsigned char block[2][sizeof(DevBlock)];
};
static_assert(sizeof(Tile) == 5 * sizeof(int) && sizeof(DevBlock) % 8 == 0 && sizeof(DevBlock) / 8 <= 64,
              "copied by one warp: a word of the tile and two words of the descriptor per lane");
__shared__ TmaShared g_tma[4];

// The compute warps' stencil source.
template <class C, bool UC>
struct TmaSource {
    static constexpr bool UNROLL = false;
    unsigned ring0;  // shared address of the ring
    const TmaShared& sh;
    unsigned full0, empty0;
    const StencilCoef& coef;  // UC: the coefficients of every block of the launch, in the kernel arguments
    unsigned int* err;
    int lin = 0;
    ArmOffsets arm{};
    int round = 0;
    int slot = 0;        // ring slot of the next field
    unsigned phase = 0;  // and the parity of its phase
    bool failed = false;

    __device__ __forceinline__ const DevBlock& block() const {
        return *reinterpret_cast<const DevBlock*>(sh.block[round & 1]);
    }
    __device__ __forceinline__ void wait() {
        if (!failed) failed = !tma_wait(full0 + 8u * slot, phase, err);
    }
    __device__ __forceinline__ const StencilCoef& coefs() const {
        if constexpr (UC)
            return coef;
        else
            return block();
    }
    template <bool HESS, bool EXACT, bool KOSEP, typename P>
    __device__ __forceinline__ FieldDer<P> der(int /*v*/, const Advection<P, EXACT>& adv) {
        wait();
        const unsigned at = ring0 + slot * (unsigned)(C::SLOT * sizeof(double));
        const SplitLoad<C::BX, C::BX * C::BY> L{at, at + lin, arm};
        const FieldDer<P> r = field_der_l<P, HESS, true, EXACT, KOSEP>(coefs(), L, adv);
        // every lane's loads of the slot come before the warp's arrival
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(empty0 + 8u * slot);
        if (++slot == C::NBUF) slot = 0, phase ^= 1u;
        return r;
    }
};

// The tiles of one compute warpgroup in order: list entries first, first +
// stride, ..., or with SEL those of them whose flag is `want`. Warp-wide.
template <bool SEL>
struct TmaTileFinder {
    const unsigned char* flags;
    int want, ntiles, stride;
    int next;              // next list entry to look at
    int base = 0;          // SEL: entry of lane 0 of the last 32 looked at
    unsigned pending = 0;  // and those of them still to be taken
    __device__ __forceinline__ int find() {
        if constexpr (SEL) {
            while (!pending) {
                if (next >= ntiles) return -1;
                base = next;
                const long long ti = base + (long long)(threadIdx.x & 31) * stride;
                pending = __ballot_sync(0xffffffffu, ti < ntiles && flags[ti] == want);
                next = (int)min((long long)ntiles, base + 32ll * stride);
            }
            const int b = __ffs(pending) - 1;
            pending &= pending - 1;
            return base + b * stride;
        } else {
            const int t = next;
            if (t >= ntiles) return -1;
            next = ntiles - t > stride ? t + stride : ntiles;
            return t;
        }
    }
};

// One load warp: every lane takes part in the tile search, the copies of tile
// and descriptor and the waits; lane 0 issues the box loads.
template <class C, bool SEL>
__device__ __forceinline__ void tma_load_warp(int g, const DevBlock* __restrict__ blocks, const Tile* __restrict__ tiles,
                                             int ntiles, const StageArgs& A, unsigned ring0) {
    TmaShared& sh = g_tma[g];
    const int lane = threadIdx.x & 31;
    const unsigned full0 = smem_addr(sh.full), empty0 = smem_addr(sh.empty);
    constexpr int WORDS = sizeof(DevBlock) / 8;
    TmaTileFinder<SEL> finder{A.tile_prec, A.want_prec, ntiles, (int)gridDim.x * C::NWG,
                             (int)(g * gridDim.x + blockIdx.x)};
    // the tile of the coming round: its list entry, this lane's word of it and this lane's words of the descriptor
    int ti = finder.find();
    int tw = ti >= 0 && lane < 5 ? reinterpret_cast<const int*>(tiles + ti)[lane] : 0;
    unsigned long long d0 = 0, d1 = 0;
    auto load_desc = [&](int word, unsigned long long& x0, unsigned long long& x1) {
        const unsigned long long* src =
            reinterpret_cast<const unsigned long long*>(blocks + __shfl_sync(0xffffffffu, word, 0));
        x0 = src[lane];
        if (lane + 32 < WORDS) x1 = src[lane + 32];
    };
    if (ti >= 0) load_desc(tw, d0, d1);
    int slot = 0, q = 0;
    unsigned ephase = 1;               // parity of the slot's empty phase: the first pass finds the slots empty
    unsigned issued = 0, parity = 0;   // per slot: a copy was issued into it; the phases its barrier will complete, mod 2
    bool ok = true;
    for (int r = 0; ok; ++r) {
        // (all compute warps have left round r - 2: each arrived on a field of round r - 1)
        TmaTile& T = sh.tile[r & 1];
        if (lane < 5) reinterpret_cast<int*>(&T.t)[lane] = tw;
        if (lane == 5) T.index = ti;
        unsigned long long* B = reinterpret_cast<unsigned long long*>(sh.block[r & 1]);
        B[lane] = d0;
        if (lane + 32 < WORDS) B[lane + 32] = d1;
        __syncwarp();
        if (ti < 0) {  // no more tiles: the compute warps see it behind the next slot's barrier
            if ((ok = tma_wait(empty0 + 8u * slot, ephase, A.errflag)) && lane == 0) {
                mbar_arrive(full0 + 8u * slot);
                parity ^= 1u << slot;  // the slot's barrier completes one phase more than its copies
            }
            break;
        }
        const int blk = __shfl_sync(0xffffffffu, tw, 0), i0 = __shfl_sync(0xffffffffu, tw, 1),
                  j0 = __shfl_sync(0xffffffffu, tw, 2), k0 = __shfl_sync(0xffffffffu, tw, 3);
        const bool rem = C::REM && __shfl_sync(0xffffffffu, tw, 4) < 0;
        const size_t map = (size_t)(3 * blk + A.in_sel) * 128;
        const unsigned char* m = static_cast<const unsigned char*>(rem ? A.tmaps_rem : A.tmaps) + map;
        const unsigned char* ma = static_cast<const unsigned char*>(A.tmaps_arm) + map;
        const int zhi = k0 + (rem ? 2 * C::TZ : C::TZ) + 5;
        constexpr unsigned ARM = C::Boxes::ARM * sizeof(double);
        const unsigned arm = (rem ? C::BoxesRem::MAIN : C::Boxes::MAIN) * (unsigned)sizeof(double);
        const unsigned bytes = (rem ? C::BoxesRem::CELLS : C::Boxes::CELLS) * (unsigned)sizeof(double);
        ti = finder.find();
        tw = ti >= 0 && lane < 5 ? reinterpret_cast<const int*>(tiles + ti)[lane] : 0;
        for (int p = 0; p < NV; ++p) {
            if (!(ok = tma_wait(empty0 + 8u * slot, ephase, A.errflag))) break;
            // test switch: item test_withhold - 1 of the first warpgroup is never issued
            if (lane == 0 && !(A.test_withhold != 0 && q == A.test_withhold - 1 && blockIdx.x == 0 && g == 0)) {
                const unsigned bar = full0 + 8u * slot, dst = ring0 + slot * (unsigned)(C::SLOT * sizeof(double));
                const int f = FIELD_ORDER[p];
                mbar_expect_tx(bar, bytes);
                // (an interior index is also the cell, incl. ghosts, four lower)
                tma_load_box(dst, m, i0, j0, k0 + 3, f, bar);
                tma_load_box(dst + arm, ma, i0 + NG, j0 + NG, k0, f, bar);
                tma_load_box(dst + arm + ARM, ma, i0 + NG, j0 + NG, zhi, f, bar);
                issued |= 1u << slot;
                parity ^= 1u << slot;
            }
            __syncwarp();
            if (++slot == C::NBUF) slot = 0, ephase ^= 1u;
            ++q;
            if (p == NV / 2 && ti >= 0) load_desc(tw, d0, d1);
        }
    }
    // no copy into shared memory outlives the CTA: wait for the last one of every slot
    if (lane == 0)
        for (int s = 0; s < C::NBUF; ++s)
            if (issued >> s & 1u) tma_wait(full0 + 8u * s, (parity >> s & 1u) ^ 1u, A.errflag);
}

}  // namespace

template <int PM, int EPI, class C, bool SEL, bool UC>
__global__ void __launch_bounds__(C::NTHR, 1)
    ccz4_stage_tma_kernel(const DevBlock* __restrict__ blocks, const Tile* __restrict__ tiles, int ntiles,
                         const __grid_constant__ StageArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int g = threadIdx.x / C::NP;  // warpgroup
    if (threadIdx.x < C::NWG)
        for (int s = 0; s < C::NBUF; ++s) {
            mbar_init(smem_addr(&g_tma[threadIdx.x].full[s]), 1);
            mbar_init(smem_addr(&g_tma[threadIdx.x].empty[s]), C::NP / 32);  // every compute warp arrives
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
    TmaSource<C, UC> S{rings + g * RING, sh, smem_addr(sh.full), smem_addr(sh.empty), A.coef, A.errflag};
#pragma unroll 1
    for (int r = 0;; ++r) {
        S.wait();  // the round's first field, and with it the tile and its descriptor
        if (S.failed) break;
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
        if (S.failed) break;
    }
}

// Launchers of one tile set: C3 the mixed kernels (12 compute warps per SM), C2
// the FP64 ones (8). grids[pm][epi][sel]: the persistent grid, 0 = not instantiated.
template <class C3, class C2>
struct TmaKernelOps {
    template <int PM>
    using Cfg = typename std::conditional<PM == PM_MIXED, C3, C2>::type;
    // the register split needs the launch's full share: setmaxnreg.inc would wait for registers that never free up
    template <int PM, int EPI, bool SEL, bool UC>
    static cudaError_t configure_one(int nsm, int grids[3][2][2]) {
        using C = Cfg<PM>;
        auto k = ccz4_stage_tma_kernel<PM, EPI, C, SEL, UC>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e != cudaSuccess) return e;
        cudaFuncAttributes fa{};
        if ((e = cudaFuncGetAttributes(&fa, k))) return e;
        grids[PM][EPI][SEL ? 1 : 0] = fa.numRegs == C::LAUNCH_REGS ? nsm : 0;  // 0: not available
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
    static cudaError_t configure_rk(int nsm, int grids[3][2][2]) {
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
    static cudaError_t configure(int nsm, int grids[3][2][2]) {
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
