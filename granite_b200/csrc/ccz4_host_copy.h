// ccz4_host_copy.h -- copies between a caller's (pageable) buffers and the device:
// PIN_THREADS host threads move pieces of up to PIN_SLOT bytes through pinned slots.
// Host code only.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

#include "ccz4_common.cuh"

namespace granite_b200 {

constexpr int PIN_THREADS = 4;
constexpr size_t PIN_SLOT = 512 << 10;

// The pinned slots are shared by the contexts of the process (pinning memory
// takes milliseconds, as long as the copies of a small block): one set, handed
// to one call at a time and freed with the last context. A call that finds it
// in use pins a set of its own context's.
struct PinnedSet {
    std::mutex in_use;  // held by the call that copies through it
    std::mutex life;    // contexts and mem
    int contexts = 0;
    char* mem = nullptr;
};
inline PinnedSet g_pinned;

inline char* alloc_pinned() {
    void* p = nullptr;
    if (cudaHostAlloc(&p, 2 * PIN_THREADS * PIN_SLOT, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return static_cast<char*>(p);
}

// A context's part in it: the slots of the copy at hand, two per copy thread, each
// with the event of its last copy; own: the context's own set.
struct HostCopy {
    int device = 0;
    bool open = false;
    char* slots = nullptr;
    char* own = nullptr;
    cudaEvent_t ev[2 * PIN_THREADS] = {};

    void create(int dev) {
        std::lock_guard<std::mutex> life(g_pinned.life);
        device = dev;
        ++g_pinned.contexts;
        open = true;
    }
    void destroy() {
        cudaFreeHost(own);
        {
            std::lock_guard<std::mutex> life(g_pinned.life);
            if (open && --g_pinned.contexts == 0) {
                cudaFreeHost(g_pinned.mem);
                g_pinned.mem = nullptr;
            }
            open = false;
        }
        for (auto e : ev)
            if (e) cudaEventDestroy(e);
    }
};

// The staging slots of one call: the process's set, or the context's own. Where no
// memory can be pinned there are none (slots == nullptr), and the copies go
// straight from and to the caller's buffers.
class PinnedLease {
  public:
    explicit PinnedLease(HostCopy& c) : c_(c) {
        for (auto& e : c.ev)
            if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                e = nullptr;
                cudaGetLastError();
                return;
            }
        lock_ = std::unique_lock<std::mutex>(g_pinned.in_use, std::try_to_lock);
        if (lock_.owns_lock()) {
            std::lock_guard<std::mutex> life(g_pinned.life);
            if (!g_pinned.mem) g_pinned.mem = alloc_pinned();
            c.slots = g_pinned.mem;
        } else {
            if (!c.own) c.own = alloc_pinned();
            c.slots = c.own;
        }
    }
    // Every copy through the slots has been waited for, also after an error: a wait is
    // refused while another thread captures a stream in the global mode, unless
    // this thread is in the relaxed one.
    ~PinnedLease() {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        for (auto e : c_.ev)
            if (e) cudaEventSynchronize(e);
        cudaThreadExchangeStreamCaptureMode(&mode);
        c_.slots = nullptr;
    }

  private:
    HostCopy& c_;
    std::unique_lock<std::mutex> lock_;
};

// Run work(t, nt) on up to PIN_THREADS host threads (the caller's among them),
// as many as `pieces` are worth; the first CUDA error of any of them.
template <typename F>
cudaError_t on_copy_threads(const HostCopy& c, size_t pieces, F&& work) {
    const int hw = (int)std::thread::hardware_concurrency();
    const int nt = (int)std::min<size_t>(std::max<size_t>(1, pieces / 2), (size_t)std::min(PIN_THREADS, hw > 0 ? hw : 1));
    std::atomic<int> err{(int)cudaSuccess};
    auto run = [&](int t, int n) {
        cudaError_t e = cudaSetDevice(c.device);
        if (e == cudaSuccess) e = work(t, n);
        int none = (int)cudaSuccess;
        if (e != cudaSuccess) err.compare_exchange_strong(none, (int)e);
    };
    std::thread th[PIN_THREADS];
    int started = 1;
    try {
        for (; started < nt; ++started) th[started] = std::thread(run, started, nt);
    } catch (const std::exception&) {
        // no thread left (system_error) or no memory for one (bad_alloc): the caller
        // takes the rest of the shares
    }
    run(0, nt);
    for (int t = started; t < nt; ++t) run(t, nt);
    for (int t = 1; t < started; ++t) th[t].join();
    return (cudaError_t)err.load();
}

// Host buffer -> device, queued on s when it returns (the host buffer is free
// again). A copy straight from pageable memory is staged by one thread (12 GB/s).
inline cudaError_t copy_in(HostCopy& c, void* dst, const void* src, size_t bytes, cudaStream_t s) {
    if (!c.slots) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
    const size_t pieces = (bytes + PIN_SLOT - 1) / PIN_SLOT;
    return on_copy_threads(c, pieces, [&](int t, int nt) {
        for (size_t q = t, n = 0; q < pieces; q += nt, ++n) {
            const int slot = 2 * t + (int)(n & 1);
            const size_t off = q * PIN_SLOT, len = std::min(PIN_SLOT, bytes - off);
            cudaError_t e = n >= 2 ? cudaEventSynchronize(c.ev[slot]) : cudaSuccess;
            if (e != cudaSuccess) return e;
            std::memcpy(c.slots + slot * PIN_SLOT, static_cast<const char*>(src) + off, len);
            e = cudaMemcpyAsync(static_cast<char*>(dst) + off, c.slots + slot * PIN_SLOT, len, cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaEventRecord(c.ev[slot], s);
            if (e != cudaSuccess) return e;
        }
        // the slots are reused by the next copy
        for (int k = 0; k < 2; ++k) {
            const cudaError_t e = cudaEventSynchronize(c.ev[2 * t + k]);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    });
}

// The interior cells of nv fields of a block of n[] interior cells, device -> host
// (both in the block's layout; the host's ghost cells keep their values). Pieces
// are runs of rows of one plane or of whole planes.
inline cudaError_t copy_out_interior(HostCopy& c, double* dst, const double* src, const int n[3], int nv, cudaStream_t s) {
    const size_t nx = n[0], ny = n[1], nz = n[2];
    const size_t tx = nx + 2 * NG, ty = ny + 2 * NG, N = tx * ty * (nz + 2 * NG);
    const size_t row = tx * sizeof(double);
    if (!c.slots || row > PIN_SLOT) {  // nothing pinned, or no row fits a slot
        for (int v = 0; v < nv; ++v)
            for (size_t k = 0; k < nz; ++k) {
                const size_t at = v * N + ((k + NG) * ty + NG) * tx + NG;
                const cudaError_t e = cudaMemcpy2DAsync(dst + at, row, src + at, row, nx * sizeof(double), ny,
                                                        cudaMemcpyDeviceToHost, s);
                if (e != cudaSuccess) return e;
            }
        return cudaStreamSynchronize(s);
    }
    const size_t rows_per = PIN_SLOT / row;
    const size_t rows = ty * nz;                                 // of a field, from its first interior plane on
    const size_t per_field = (rows + rows_per - 1) / rows_per, pieces = per_field * nv;
    return on_copy_threads(c, pieces, [&](int t, int nt) {
        size_t first[2] = {}, count[2] = {};  // the piece in each slot
        double* base[2] = {};
        auto finish = [&](int k) {
            cudaError_t e = cudaEventSynchronize(c.ev[2 * t + k]);
            if (e != cudaSuccess) return e;
            for (size_t q = 0; q < count[k]; ++q) {
                const size_t j = (first[k] + q) % ty;
                if (j < NG || j >= NG + ny) continue;
                std::memcpy(base[k] + (first[k] + q) * tx + NG,
                            reinterpret_cast<const double*>(c.slots + (2 * t + k) * PIN_SLOT) + q * tx + NG,
                            nx * sizeof(double));
            }
            return cudaSuccess;
        };
        size_t m = 0;
        for (size_t p = t; p < pieces; p += nt, ++m) {
            const int k = (int)(m & 1);
            cudaError_t e = m >= 2 ? finish(k) : cudaSuccess;
            if (e != cudaSuccess) return e;
            const size_t v = p / per_field;
            first[k] = (p % per_field) * rows_per;
            count[k] = std::min(rows_per, rows - first[k]);
            const size_t origin = v * N + (size_t)NG * tx * ty;
            base[k] = dst + origin;
            e = cudaMemcpyAsync(c.slots + (2 * t + k) * PIN_SLOT, src + origin + first[k] * tx, count[k] * row,
                                cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaEventRecord(c.ev[2 * t + k], s);
            if (e != cudaSuccess) return e;
        }
        for (size_t q = m > 2 ? m - 2 : 0; q < m; ++q) {
            const cudaError_t e = finish((int)(q & 1));
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    });
}

}  // namespace granite_b200
