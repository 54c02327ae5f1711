// The staged copies of the host-buffer operator (ccz4_host_copy.h) over a fake
// runtime whose "device" is host memory: with slots, where no memory can be
// pinned, where no event can be made, and where a thread cannot be started (none
// left, or no memory for its state), for blocks of one piece, of many with a
// ragged last one, and of rows wider than a slot.
#include <dlfcn.h>
#include <pthread.h>

#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "ccz4_host_copy.h"

static std::atomic<bool> copying{false};                            // within a copy:
static bool no_threads = false, no_thread_state = false;  // what fails there

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) noexcept {
    static const auto real = reinterpret_cast<decltype(&pthread_create)>(dlsym(RTLD_NEXT, "pthread_create"));
    return copying && no_threads ? EAGAIN : real(t, a, f, x);
}
void* operator new(size_t n) {
    if (void* p = copying && no_thread_state ? nullptr : std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static bool no_pinned = false, no_events = false, no_copies = false;
static bool capturing = false;  // another thread captures a stream in the global mode
static thread_local cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
static int pinned = 0, events = 0;
static std::mutex in_flight_m;
static std::set<cudaEvent_t> in_flight;  // recorded and not waited for

cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (no_pinned) return cudaErrorMemoryAllocation;
    ++pinned;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    if (p) --pinned;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    if (no_events) return cudaErrorMemoryAllocation;
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    ++events;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    --events;
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    std::lock_guard<std::mutex> l(in_flight_m);
    const bool was = copying;
    copying = false;  // (the set's own memory)
    in_flight.insert(e);
    copying = was;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (capturing && mode != cudaStreamCaptureModeRelaxed) return cudaErrorInvalidValue;
    std::lock_guard<std::mutex> l(in_flight_m);
    in_flight.erase(e);
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
    std::swap(*m, mode);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (no_copies) return cudaErrorInvalidValue;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    if (no_copies) return cudaErrorInvalidValue;
    for (size_t r = 0; r < h; ++r) std::memcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

using namespace granite_b200;

static int round_trip(const int n[3], int nv) {
    const size_t tx = n[0] + 2 * NG, ty = n[1] + 2 * NG, tz = n[2] + 2 * NG, N = tx * ty * tz;
    std::vector<double> u(nv * N), dev(nv * N, -1.0), back(nv * N, -2.0);
    for (size_t k = 0; k < u.size(); ++k) u[k] = (double)k;
    HostCopy c;
    c.create(0);
    int bad = 0;
    for (int again = 0; again < 2; ++again) {
        PinnedLease lease(c);
        copying = true;
        bad += copy_in(c, dev.data(), u.data(), u.size() * sizeof(double), nullptr) != cudaSuccess;
        bad += copy_out_interior(c, back.data(), dev.data(), n, nv, nullptr) != cudaSuccess;
        copying = false;
    }
    bad += dev != u;
    auto inner = [&](size_t i, int d) { return i >= (size_t)NG && i < (size_t)(NG + n[d]); };
    for (size_t k = 0; k < back.size(); ++k) {
        const size_t q = k % N;
        const bool in = inner(q % tx, 0) && inner(q / tx % ty, 1) && inner(q / (tx * ty), 2);
        bad += back[k] != (in ? u[k] : -2.0);
    }
    c.destroy();
    return bad + (pinned != 0) + (events != 0);
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    no_pinned = what == "no_pinned";
    no_events = what == "no_events";
    no_threads = what == "no_threads";
    no_thread_state = what == "no_thread_state";
    const int small[3] = {5, 3, 2}, many[3] = {64, 40, 33}, wide[3] = {65600, 2, 1};
    int bad = round_trip(small, 22) + round_trip(many, 22) + round_trip(wide, 2);
    if (what == "copy_error") {  // an error of a copy is the call's
        no_copies = true;
        std::vector<double> a(1 << 20), b(1 << 20);
        HostCopy c;
        c.create(0);
        {
            PinnedLease lease(c);
            bad += copy_in(c, b.data(), a.data(), a.size() * sizeof(double), nullptr) == cudaSuccess;
            bad += copy_out_interior(c, b.data(), a.data(), small, 22, nullptr) == cudaSuccess;
        }
        c.destroy();
    }
    if (what == "capture_elsewhere") {  // the call fails, but hands the slots on with no copy in flight
        capturing = true;
        std::vector<double> a(1 << 20), b(1 << 20);
        HostCopy c;
        c.create(0);
        {
            PinnedLease lease(c);
            bad += copy_in(c, b.data(), a.data(), a.size() * sizeof(double), nullptr) == cudaSuccess;
            bad += in_flight.empty();
        }
        bad += !in_flight.empty() || mode != cudaStreamCaptureModeGlobal;
        c.destroy();
    }
    std::printf(bad ? "%d wrong\n" : "OK\n", bad);
    return bad != 0;
}
