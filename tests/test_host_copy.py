"""Which way a large result takes to the host (csrc/host_copy.h), with a fake of the
CUDA calls that the header makes: pageable destinations through the pinned buffers,
pinned ones and those where the buffers or the threads run out by what is left, always
the same bytes and nothing outside the rows."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "titus_b200", "csrc")

FAKE = r"""
#pragma once
#include <atomic>
#include <cstdlib>
#include <cstring>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum { cudaMemcpyDeviceToHost, cudaHostAllocPortable, cudaStreamNonBlocking, cudaEventDisableTiming };
typedef int* cudaStream_t;
typedef int* cudaEvent_t;
struct cudaPointerAttributes { cudaMemoryType type; };
struct Fake {
    std::atomic<int> plain{0}, staged{0};
    bool pinned = false, no_pool = false;
    int threads_left = 1 << 20;
};
inline Fake fake;
inline int handle_;
inline void rows(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h) {
    for (size_t r = 0; r < h; ++r) memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
}
inline cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, int) {
    ++fake.plain;
    rows(d, dp, s, sp, w, h);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t) {
    ++fake.staged;
    memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, int, cudaStream_t) {
    ++fake.staged;
    rows(d, dp, s, sp, w, h);
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    a->type = fake.pinned ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, int) {
    if (fake.no_pool) return cudaErrorMemoryAllocation;
    *p = malloc(n);
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, int) { *s = &handle_; return cudaSuccess; }
inline cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = &handle_; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
"""

MAIN = r"""
#include <dlfcn.h>
#include <cerrno>
#include <cstdio>
#include <pthread.h>
#include <vector>
#include "host_copy.h"

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) noexcept {
    if (fake.threads_left-- <= 0) return EAGAIN;
    static auto real = (int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*))dlsym(RTLD_NEXT, "pthread_create");
    return real(t, a, f, x);
}

// h rows of w doubles, from rows of sp into rows of dp
static int check(const char* what, size_t w, size_t sp, size_t dp, size_t h, bool staged, bool fresh = false) {
    std::vector<double> src(sp * h);
    auto* dst = (double*)mmap(nullptr, dp * h * 8, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (!fresh) std::fill_n(dst, dp * h, 7.5);
    for (size_t i = 0; i < src.size(); ++i) src[i] = (double)i;
    titus_host::HostCopy copy;
    fake.plain = fake.staged = 0;
    const int rc = copy.copy2d(dst, dp * 8, src.data(), sp * 8, w * 8, h);
    copy.release();
    bool same = rc == 0;
    for (size_t r = 0; r < h && same; ++r)
        for (size_t j = 0; j < dp && same; ++j) same = dst[r * dp + j] == (j < w ? src[r * sp + j] : 7.5);
    munmap(dst, dp * h * 8);
    const bool way = staged ? fake.plain == 0 && fake.staged > 0 : fake.plain == 1 && fake.staged == 0;
    if (!same || !way) printf("%s: rc %d, bytes %s, %d plain, %d staged\n", what, rc, same ? "equal" : "differ",
                              (int)fake.plain, (int)fake.staged);
    return !(same && way);
}
int main() {
    const bool lanes = std::thread::hardware_concurrency() > 1;
    int bad = check("small", 19, 80, 80, 1000, false);
    bad += check("strided", 19, 80, 80, 40001, lanes);
    bad += check("contiguous, pages there", 900, 900, 900, 4503, false);
    bad += check("contiguous, fresh pages", 900, 900, 900, 4503, lanes, true);
    bad += check("contiguous from strided rows, fresh pages", 20, 24, 20, 220001, lanes, true);
    bad += check("contiguous, pages there, 144 MB", 900, 900, 900, 20003, lanes);
    bad += check("wide rows", 40000, 40000, 40000, 57, false);
    fake.threads_left = 2;
    bad += check("two more threads", 19, 80, 80, 40001, lanes);
    fake.threads_left = 0;
    bad += check("no more threads", 900, 900, 900, 4503, lanes, true);
    fake.threads_left = 1 << 20;
    fake.no_pool = true;
    bad += check("no buffers", 19, 80, 80, 40001, false);
    fake.no_pool = false;
    fake.pinned = true;
    bad += check("pinned, strided", 19, 80, 80, 40001, false);
    bad += check("pinned, contiguous", 900, 900, 900, 20003, false);
    return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_ways_to_the_host(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "host_copy")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(tmp_path), "-I", CSRC, "-o", exe,
                    str(tmp_path / "main.cpp"), "-ldl"], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
