// Device-to-host copies of large results into pageable memory.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

namespace titus_host {

// cudaMemcpy2D to pageable memory goes through one thread, which takes every page
// fault of a fresh result array and copies row by row (40 000 rows of 19 values
// into rows of 80: 20 ms; 40 000 x 900 contiguous: 78 ms, 18 when the pages are
// there). Here up to kThreads threads take a span of the rows each and copy it by
// chunks through two pinned buffers of their own, one chunk in flight while the
// other is scattered. Spans, not chunks dealt in turn: threads that write to one
// huge page fault it together, and 6 MB of fresh contiguous rows then took 5 to 11
// ms instead of 0.4. The buffers (4 MiB in all), streams
// and the events are made by the first large copy of a handle and freed with it.
// From kLarge bytes of destination on (32 MB into fresh pages: strided 26 -> 1.9 ms,
// contiguous 14 -> 2.6; into touched ones 16.5 -> 0.7 and 2.0 -> 1.7). 8 MB of strided
// rows would gain as well when repeated (6.1 -> 1.2 ms), but a handle's first copy,
// which makes the buffers, costs 5 ms and more, and counts as much.
// Pinned (and managed) destinations keep the plain copy: the engine writes them directly
// (288 MB contiguous: 5.1 ms, 14.4 through the buffers; 160 000 rows of 20 values into
// rows of 80: 0.64 and 2.2; 40 000 of 2 into 80: 0.10 and 0.3).
// So do contiguous destinations below kDense whose pages are there, where one thread has
// nothing to fault in and no rows to deal with (17 MB: 0.92 ms, 1.1 through the buffers;
// 24 MB 1.3 and 1.6; 66 MB 3.4 and 3.6; 117 MB 6.1 and 6.3; 288 MB 15.6 and 14.4).
// Device work that writes the source must have completed.
class HostCopy {
public:
    static constexpr int kThreads = 8;
    static constexpr size_t kChunk = 256u << 10, kSpan = 2u << 20, kLarge = 16u << 20, kDense = 128u << 20;

    // the row-wise copy of cudaMemcpy2D(..., cudaMemcpyDeviceToHost), pitches in bytes
    cudaError_t copy2d(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, size_t height) {
        const size_t bytes = height * dpitch;
        if (bytes < kLarge || width == 0 || width > kChunk || !pageable(dst) ||
            (dpitch == width && bytes < kDense && resident(dst, bytes)))
            return cudaMemcpy2D(dst, dpitch, src, spitch, width, height, cudaMemcpyDeviceToHost);
        std::lock_guard<std::mutex> hold(lock_);
        const int nt = lanes((int)std::min<size_t>(kThreads, bytes / kSpan));
        if (nt < 2) return cudaMemcpy2D(dst, dpitch, src, spitch, width, height, cudaMemcpyDeviceToHost);
        int device = 0;
        cudaError_t rc = cudaGetDevice(&device);
        if (rc != cudaSuccess) return rc;
        const size_t rows = kChunk / width, span = (height + nt - 1) / nt;
        std::atomic<int> part{0};
        std::atomic<int> err{(int)cudaSuccess};
        const auto work = [&](Lane* L) {
            cudaError_t e = cudaSetDevice(device);
            for (int p; (p = part.fetch_add(1)) < nt && e == cudaSuccess;) {
                const size_t end = std::min(height, (p + 1) * span);
                size_t next = std::min(height, p * span), at[2] = {end, end};
                const auto fetch = [&](int b) {
                    at[b] = next;
                    if (next == end || e != cudaSuccess) return;
                    const size_t n = std::min(rows, end - next);
                    const char* s = static_cast<const char*>(src) + next * spitch;
                    next += n;
                    e = spitch == width ? cudaMemcpyAsync(L->buf[b], s, n * width, cudaMemcpyDeviceToHost, L->stream)
                                        : cudaMemcpy2DAsync(L->buf[b], width, s, spitch, width, n, cudaMemcpyDeviceToHost,
                                                            L->stream);
                    if (e == cudaSuccess) e = cudaEventRecord(L->done[b], L->stream);
                };
                fetch(0);
                for (int b = 0; at[b] < end && e == cudaSuccess; b ^= 1) {
                    fetch(b ^ 1);
                    if (e == cudaSuccess) e = cudaEventSynchronize(L->done[b]);
                    if (e != cudaSuccess) break;
                    const size_t n = std::min(rows, end - at[b]);
                    char* d = static_cast<char*>(dst) + at[b] * dpitch;
                    if (dpitch == width) {
                        std::memcpy(d, L->buf[b], n * width);
                    } else {
                        for (size_t r = 0; r < n; ++r) std::memcpy(d + r * dpitch, L->buf[b] + r * width, width);
                    }
                    at[b] = end;
                }
            }
            if (e != cudaSuccess) {
                cudaStreamSynchronize(L->stream);   // nothing in flight into the buffers
                err.store((int)e);
            }
        };
        std::thread th[kThreads - 1];
        int started = 0;
        try {
            for (; started < nt - 1; ++started) th[started] = std::thread(work, &lane_[started + 1]);
        } catch (...) {   // no more threads: those that run, and this one, take all rows
        }
        work(&lane_[0]);
        for (int t = 0; t < started; ++t) th[t].join();
        return (cudaError_t)err.load();
    }

    void release() {
        for (Lane& L : lane_)
            for (int b = 0; b < 2; ++b)
                if (L.done[b]) cudaEventDestroy(L.done[b]);
        for (cudaStream_t& st : stream_) {
            if (st) cudaStreamDestroy(st);
            st = nullptr;
        }
        if (pinned_) cudaFreeHost(pinned_);
        for (Lane& L : lane_) L = Lane{};
        pinned_ = nullptr;
        ready_ = false;
    }

private:
    struct Lane {
        cudaEvent_t done[2] = {nullptr, nullptr};
        char* buf[2] = {nullptr, nullptr};
        cudaStream_t stream = nullptr;
    };
    Lane lane_[kThreads];
    cudaStream_t stream_[2] = {nullptr, nullptr};   // of the even and the odd lanes: two keep the copy engines busy
    char* pinned_ = nullptr;
    bool ready_ = false;
    std::mutex lock_;

    static bool pageable(const void* p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
        cudaGetLastError();
        return false;
    }
    // the pages at three places inside: the first one can be there by its allocator's header alone
    static bool resident(const void* p, size_t bytes) {
        const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
        for (int part = 1; part < 4; ++part) {
            const uintptr_t at = ((uintptr_t)p + bytes / 4 * part) / page * page;
            unsigned char in = 0;
            if (mincore((void*)at, page, &in) == 0 && !(in & 1)) return false;
        }
        return true;
    }
    // the lanes that can be used: none (the plain copy serves) when something runs out
    int lanes(int want) {
        want = (int)std::min<unsigned>(want, std::max(1u, std::thread::hardware_concurrency()));
        if (want < 2) return 0;
        if (!ready_ && !make()) {
            cudaGetLastError();
            release();
            return 0;
        }
        ready_ = true;
        return want;
    }
    bool make() {
        if (cudaHostAlloc((void**)&pinned_, kThreads * 2 * kChunk, cudaHostAllocPortable) != cudaSuccess) return false;
        for (cudaStream_t& st : stream_)
            if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return false;
        for (int t = 0; t < 2 * kThreads; ++t) {
            Lane& L = lane_[t / 2];
            L.buf[t % 2] = pinned_ + t * kChunk;
            L.stream = stream_[(t / 2) % 2];
            if (cudaEventCreateWithFlags(&L.done[t % 2], cudaEventDisableTiming) != cudaSuccess) return false;
        }
        return true;
    }
};

}  // namespace titus_host
