// ccz4_stage_ring.cuh -- the field ring of the TMA stage kernel: the tiles and
// barriers in shared memory, the load warps and the compute warps' waits.
//
// Only the protocol: the includer provides the primitives it is written with
// (smem_addr, mbar_expect_tx, mbar_try_wait, mbar_arrive, global_ns,
// tma_load_box) and FIELD_ORDER. The kernel's are PTX (ccz4_stage_tma.cuh); the
// CPU test of the protocol has its own.
#pragma once

#include "ccz4_common.cuh"

namespace granite_b200 {

namespace {

// Wait limit of one ring slot: 2 s of wall time, then the kernel records the
// failure in StageArgs::errflag and stops waiting (results are then garbage
// and the host reports the error).
constexpr unsigned long long TMA_WAIT_NS = 2000000000ull;

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
    int stop;  // 1: a compute lane's wait ran out
    TmaTile tile[2];
    __align__(16) unsigned char block[2][sizeof(DevBlock)];
};
static_assert(sizeof(Tile) == 5 * sizeof(int) && sizeof(DevBlock) % 8 == 0 && sizeof(DevBlock) / 8 <= 64,
              "copied by one warp: a word of the tile and two words of the descriptor per lane");
__shared__ TmaShared g_tma[4];

// One compute warp's side of its warpgroup's ring, lane by lane. A lane whose wait
// ran out waits no more (what it reads then is within the slot, and dropped with
// the launch) and stops the load warp: a slot it gave up on may have a copy in
// flight, and no other may be issued into it. The warp leaves together at the next
// round. (The flag and the one vote a round keep this out of the field loop; with
// a vote in every wait the steps of a 3-level hierarchy took 0.8 % longer.)
template <int NBUF>
struct TmaRing {
    TmaShared& sh;
    unsigned full0, empty0;  // shared addresses of sh.full and sh.empty
    unsigned int* err;
    int slot = 0;        // ring slot of the next field
    unsigned phase = 0;  // and the parity of its phase
    bool failed = false;

    __device__ __forceinline__ void wait() {
        if (!failed && !tma_wait(full0 + 8u * slot, phase, err)) {
            failed = true;
            *const_cast<volatile int*>(&sh.stop) = 1;  // (before the warp's next arrival)
        }
    }
    // Wait for a round's first field, and with it the tile and its descriptor;
    // false: a wait of the warp ran out.
    __device__ __forceinline__ bool next_round() {
        wait();
        return __all_sync(0xffffffffu, !failed);
    }
    __device__ __forceinline__ void release() {
        // every lane's loads of the slot come before the warp's arrival
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(empty0 + 8u * slot);
        if (++slot == NBUF) slot = 0, phase ^= 1u;
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
// and descriptor and the waits; lane 0 issues the box loads. A wait that ran out
// in one lane, of this warp or of a compute warp (TmaShared::stop), ends the loop
// for all of them: lanes left behind would read lane 0's words after it is gone.
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
    auto slot_empty = [&]() {
        const bool e = tma_wait(empty0 + 8u * slot, ephase, A.errflag);
        return __all_sync(0xffffffffu, e && !*const_cast<const volatile int*>(&sh.stop)) != 0;
    };
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
            ok = slot_empty();
            if (ok && lane == 0) {
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
            if (!(ok = slot_empty())) break;
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
    // no copy into shared memory outlives the CTA: wait for the last one of every
    // slot (the one before it has landed: every compute lane saw it)
    if (lane == 0)
        for (int s = 0; s < C::NBUF; ++s)
            if (issued >> s & 1u) tma_wait(full0 + 8u * s, (parity >> s & 1u) ^ 1u, A.errflag);
}

}  // namespace

}  // namespace granite_b200
