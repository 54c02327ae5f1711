// The ring protocol of the TMA stage kernel (ccz4_stage_ring.cuh) on host
// threads, one per lane: a load warp and the four compute warps of a warpgroup,
// with emulated barriers, warp collectives and copies. Checked in every run:
//   * a warp collective is entered by all 32 lanes (a lane that left the code
//     around it would be a read of an inactive lane on the device);
//   * no copy is issued into a slot whose previous copy is in flight;
//   * no copy is in flight when the last warp has left.
// Waits that run out are made with the clock of single lanes, so that some
// lanes of a warp give up where others succeed.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "ccz4_common.cuh"

using Clock = std::chrono::steady_clock;

[[noreturn]] static void violation(const char* what) {
    std::printf("violation: %s\n", what);
    std::fflush(stdout);
    std::_Exit(1);
}

// ---- lanes and warps ----------------------------------------------------------

struct Warp {
    std::mutex m;
    std::condition_variable cv;
    int in = 0, gone = 0;
    long long generation = 0;
    int value[32] = {};
    int result[32] = {};
    // every lane's value, once all 32 are in
    void all(int lane, int v, int out[32]) {
        std::unique_lock<std::mutex> l(m);
        if (gone) violation("warp collective without all lanes");
        value[lane] = v;
        if (++in == 32) {
            in = 0;
            ++generation;
            std::memcpy(result, value, sizeof(value));
            cv.notify_all();
        } else {
            const long long g = generation;
            if (!cv.wait_for(l, std::chrono::seconds(20), [&] { return generation != g || gone; }))
                violation("warp collective not entered by every lane");
            if (generation == g) violation("warp collective without all lanes");
        }
        std::memcpy(out, result, sizeof(result));
    }
    void leave() {
        std::lock_guard<std::mutex> l(m);
        ++gone;
        cv.notify_all();
    }
};

struct Dim {
    unsigned x;
};
static thread_local Dim threadIdx{0};
static thread_local Warp* t_warp = nullptr;
static thread_local long long t_skew = 0;  // ns added to this lane's clock at every look,
static std::atomic<bool> g_skewed{false};  // once the run has come to the wait in question
static Dim blockIdx{0}, gridDim{1};

static int lane() { return threadIdx.x & 31; }
template <typename T>
static T __shfl_sync(unsigned, T v, int from) {
    int out[32];
    t_warp->all(lane(), (int)v, out);
    return (T)out[from];
}
static unsigned __ballot_sync(unsigned, bool p) {
    int out[32];
    t_warp->all(lane(), p, out);
    unsigned b = 0;
    for (int k = 0; k < 32; ++k) b |= out[k] ? 1u << k : 0u;
    return b;
}
static bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == 0xffffffffu; }
static void __syncwarp() { __ballot_sync(0xffffffffu, true); }
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
static std::atomic<unsigned> g_err{0};
static void atomicExch(unsigned*, unsigned v) { g_err = v; }
using std::min;

// ---- barriers and copies --------------------------------------------------------

namespace granite_b200 {
namespace {
constexpr int FIELD_ORDER[NV] = {1, 2, 3, 4, 5, 6, 14, 15, 16, 0, 18, 19, 20, 21, 13, 17, 7, 8, 9, 10, 11, 12};
inline unsigned smem_addr(const void* p);
void mbar_expect_tx(unsigned bar, unsigned bytes);
bool mbar_try_wait(unsigned bar, unsigned parity);
void mbar_arrive(unsigned bar);
unsigned long long global_ns();
void tma_load_box(unsigned dst, const void* map, int x, int y, int z, int f, unsigned bar);
}  // namespace
}  // namespace granite_b200

#include "ccz4_stage_ring.cuh"

namespace granite_b200 {
namespace {

struct Bar {
    int count = 0, pending = 0;
    long long tx = 0;
    unsigned phase = 0;
    void check() {
        if (pending == 0 && tx == 0) {
            ++phase;
            pending = count;
        }
    }
};
struct Copy {
    unsigned dst, bar, bytes;
    int x, y, z, f;
    Clock::time_point due;
};
struct Smem {
    std::mutex m;
    std::map<unsigned, Bar> bars;
    std::vector<Copy> flying;
    std::vector<Copy> issued;
    std::function<int(long long)> delay_ms = [](long long) { return 0; };  // of the n-th box
    bool quit = false;
} g_mem;

inline unsigned smem_addr(const void* p) { return (unsigned)((const char*)p - (const char*)&g_tma[0]); }
unsigned long long global_ns() {
    static thread_local long long skew = 0;
    if (g_skewed) skew += t_skew;
    return (unsigned long long)(std::chrono::duration_cast<std::chrono::nanoseconds>(Clock::now().time_since_epoch()).count() + skew);
}
Bar& bar_of(unsigned b) {
    const auto it = g_mem.bars.find(b);
    if (it == g_mem.bars.end()) violation("no such barrier");
    return it->second;
}
void mbar_expect_tx(unsigned b, unsigned bytes) {
    std::lock_guard<std::mutex> l(g_mem.m);
    Bar& r = bar_of(b);
    if (r.pending == 0) violation("barrier armed twice in a phase");
    r.tx += bytes;
    --r.pending;
    r.check();
}
void mbar_arrive(unsigned b) {
    std::lock_guard<std::mutex> l(g_mem.m);
    Bar& r = bar_of(b);
    if (r.pending == 0) violation("more arrivals than a phase has");
    --r.pending;
    r.check();
}
bool mbar_try_wait(unsigned b, unsigned parity) {
    {
        std::lock_guard<std::mutex> l(g_mem.m);
        if ((bar_of(b).phase & 1u) != parity) return true;
    }
    std::this_thread::sleep_for(std::chrono::microseconds(100));
    return false;
}

// ---- the kernel of the test -----------------------------------------------------

struct TestKernel {  // the shapes of TmaKernelT; slot addresses need no storage here
    static constexpr int NWG = 1, NBUF = 3, TZ = 2, SLOT = 1024;
    static constexpr bool REM = true;
    struct Boxes {
        static constexpr int MAIN = 600, ARM = 100, CELLS = MAIN + 2 * ARM;
    };
    struct BoxesRem {
        static constexpr int MAIN = 800, ARM = 100, CELLS = MAIN + 2 * ARM;
    };
};
using C = TestKernel;
constexpr unsigned SLOTS = 1u << 20;  // address of the ring's slots
unsigned char g_maps[3][3 * 128 * 4];  // main, remainder and far-plane maps of 4 blocks

void tma_load_box(unsigned dst, const void* map, int x, int y, int z, int f, unsigned bar) {
    const auto in = [&](int k) { return map >= g_maps[k] && map < g_maps[k] + sizeof(g_maps[k]); };
    if (!in(0) && !in(1) && !in(2)) violation("tensor map out of range");
    const unsigned bytes = (in(0) ? C::Boxes::MAIN : in(1) ? C::BoxesRem::MAIN : C::Boxes::ARM) * sizeof(double);
    std::lock_guard<std::mutex> l(g_mem.m);
    const unsigned slot = (dst - SLOTS) / (C::SLOT * sizeof(double));
    for (const Copy& c : g_mem.flying)
        if (c.bar != bar ? (c.dst - SLOTS) / (C::SLOT * sizeof(double)) == slot : c.dst == dst)
            violation("copy into a slot whose previous copy is in flight");
    const Copy c{dst, bar, bytes, x, y, z, f,
                 Clock::now() + std::chrono::milliseconds(g_mem.delay_ms((long long)g_mem.issued.size()))};
    g_mem.flying.push_back(c);
    g_mem.issued.push_back(c);
}
void copy_engine() {
    for (;;) {
        {
            std::lock_guard<std::mutex> l(g_mem.m);
            const auto now = Clock::now();
            for (size_t k = 0; k < g_mem.flying.size();) {
                if (g_mem.flying[k].due > now) {
                    ++k;
                    continue;
                }
                const Copy c = g_mem.flying[k];
                g_mem.flying.erase(g_mem.flying.begin() + (long)k);
                Bar& r = bar_of(c.bar);
                r.tx -= c.bytes;
                r.check();
            }
            if (g_mem.quit) return;
        }
        std::this_thread::sleep_for(std::chrono::microseconds(50));
    }
}

std::vector<Tile> g_tiles;
std::vector<DevBlock> g_blocks;
std::vector<unsigned char> g_flags;
std::function<void(int warp, int round, int field)> g_at_field = [](int, int, int) {};
std::function<long long(int warp, int lane)> g_skew = [](int, int) { return 0ll; };  // warp -1: the load warp
std::mutex g_seen_m;
std::map<int, int> g_seen;  // list entry -> lanes that went through it

// The loop of the kernel's compute warps, without the arithmetic.
void compute_lane(int warp, const StageArgs& A) {
    TmaRing<C::NBUF> ring{g_tma[0], smem_addr(g_tma[0].full), smem_addr(g_tma[0].empty), A.errflag};
    for (int r = 0;; ++r) {
        if (!ring.next_round()) break;
        const int ti = g_tma[0].tile[r & 1].index;
        if (ti < 0) break;
        {
            std::lock_guard<std::mutex> l(g_seen_m);
            ++g_seen[ti];
        }
        DevBlock B;
        std::memcpy(&B, g_tma[0].block[r & 1], sizeof(B));
        if (B.level != g_tma[0].tile[r & 1].t.block) violation("descriptor of another block");
        for (int f = 0; f < NV; ++f) {
            ring.wait();
            g_at_field(warp, r, f);
            ring.release();
        }
        // (a failed warp's epilogue reads the round's tile and descriptor too)
        if (g_tma[0].tile[r & 1].index != ti) violation("tile of a round overwritten before its end");
    }
}

template <bool SEL>
void run(int ntiles) {
    StageArgs A{};
    A.tmaps = g_maps[0];
    A.tmaps_rem = g_maps[1];
    A.tmaps_arm = g_maps[2];
    unsigned errflag = 0;
    A.errflag = &errflag;
    if (SEL) A.tile_prec = g_flags.data(), A.want_prec = 1;
    for (int s = 0; s < C::NBUF; ++s) {
        g_mem.bars[smem_addr(&g_tma[0].full[s])] = Bar{1, 1, 0, 0};
        g_mem.bars[smem_addr(&g_tma[0].empty[s])] = Bar{4, 4, 0, 0};
    }
    Warp warps[5];
    std::vector<std::thread> lanes;
    std::thread engine(copy_engine);
    for (int w = 0; w < 5; ++w)
        for (int l = 0; l < 32; ++l)
            lanes.emplace_back([&, w, l] {
                t_warp = &warps[w];
                threadIdx.x = (unsigned)(32 * w + l);
                t_skew = g_skew(w < 4 ? w : -1, l);
                if (w < 4)
                    compute_lane(w, A);
                else
                    tma_load_warp<C, SEL>(0, g_blocks.data(), g_tiles.data(), ntiles, A, SLOTS);
                t_warp->leave();
            });
    for (auto& t : lanes) t.join();
    std::lock_guard<std::mutex> l(g_mem.m);
    if (!g_mem.flying.empty()) violation("copy in flight after the last warp left");
    g_mem.quit = true;
    engine.detach();
}

}  // namespace
}  // namespace granite_b200

using namespace granite_b200;

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const int n = 7;
    for (int b = 0; b < 4; ++b) {
        DevBlock d{};
        d.level = b;
        g_blocks.push_back(d);
    }
    for (int t = 0; t < 40; ++t) {
        g_tiles.push_back(Tile{t % 4, 16 * t, 4 * t, 2 * t, t % 3 == 2 ? -8 : 0});
        g_flags.push_back(t % 5 == 1);
    }
    const long long LATE = 3000000000ll;  // a lane whose clock jumps past the wait limit at its second look
    bool expect_error = true;
    if (what == "tiles" || what == "selected") {  // no wait runs out: every tile once, every box where it belongs
        const bool sel = what == "selected";
        if (sel)
            run<true>((int)g_tiles.size());
        else
            run<false>(n);
        std::vector<int> want;
        for (int t = 0; t < (sel ? (int)g_tiles.size() : n); ++t)
            if (!sel || g_flags[(size_t)t]) want.push_back(t);
        if (g_seen.size() != want.size()) violation("number of tiles");
        for (int t : want)
            if (g_seen[t] != 128) violation("a tile not seen by every lane");
        if (g_mem.issued.size() != want.size() * NV * 3) violation("number of boxes");
        size_t k = 0;
        for (int t : want)
            for (int f = 0; f < NV; ++f)
                for (int b = 0; b < 3; ++b, ++k) {
                    const Copy& c = g_mem.issued[k];
                    const Tile& tl = g_tiles[(size_t)t];
                    const int zhi = tl.k0 + (tl.w < 0 ? 4 : 2) + 5;
                    if (c.f != FIELD_ORDER[f] || c.x != tl.i0 + (b ? 4 : 0) || c.y != tl.j0 + (b ? 4 : 0) ||
                        c.z != (b == 0 ? tl.k0 + 3 : b == 1 ? tl.k0 : zhi))
                        violation("box coordinates");
                }
        expect_error = false;
    } else if (what == "load_lane_late") {  // one lane of the load warp gives up on a slot the others find empty
        g_at_field = [](int warp, int r, int f) {
            if (warp != 2 || r != 1 || f != 4) return;
            g_skewed = true;
            std::this_thread::sleep_for(std::chrono::milliseconds(300));
        };
        const int late = argc > 2 ? std::atoi(argv[2]) : 0;
        g_skew = [=](int w, int l) { return w < 0 && l == late ? LATE : 0; };
        run<false>(n);
    } else if (what == "compute_lane_late") {  // one lane of a compute warp gives up on a field the others get
        g_mem.delay_ms = [](long long box) {
            if (box / 3 != NV + 6) return 0;
            g_skewed = true;
            return 300;
        };
        const int late = argc > 2 ? std::atoi(argv[2]) : 0;
        g_skew = [=](int w, int l) { return w == 1 && l == late ? LATE : 0; };
        run<false>(n);
    } else if (what == "compute_warps_late") {  // all compute lanes give up on a field whose copy is still coming
        const int item = argc > 2 ? std::atoi(argv[2]) : 0;
        g_mem.delay_ms = [=](long long box) {
            if (box / 3 != item) return 0;
            g_skewed = true;
            return 1500;
        };
        g_skew = [=](int w, int) { return w >= 0 ? LATE : 0; };
        run<false>(n);
    } else {
        std::printf("unknown run\n");
        return 2;
    }
    if ((g_err != 0) != expect_error) violation("error flag");
    std::printf("OK\n");
    return 0;
}
