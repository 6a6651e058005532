// bdc_hostcopy.cu -- vectors of representatives from the device into pageable
// host memory.
//
// The driver copies into pageable memory through one pinned buffer on the
// calling thread.  Where the caller's pages are resident that is the fastest
// way; a large result buffer fresh from the allocator is not, and then the
// copy is mostly its page faults.  For those a few threads each take every
// n-th piece of 128 KB through two pinned buffers of their own, one being
// filled by the DMA engine while the other is copied, so that the page faults
// run in parallel.  Everything else goes the driver's way.
#include <algorithm>
#include <cstring>
#include <exception>
#include <new>
#include <thread>

#include <sched.h>
#include <sys/mman.h>
#include <unistd.h>

#include "bdc_engine.cuh"

namespace bdc {

// Milliseconds of a copy to the host, the driver's way / by the threads (16
// cores; 4.2, 8.4, 16.8, 33.6 and 67 MB):
//   resident pages   0.27/0.34  0.47/0.64  0.88/1.3  1.7/2.5  3.4/4.9
//   fresh pages       1.9/-      3.7/-      7.3/1.7  14.6/3.3  29/6.1
//   from numpy.empty    -          -          -       7.4/2.8  13.7/5.5
// A handle's first copy by the threads takes 1.2 to 2.2 ms longer (it pins the
// buffers): fresh pages 3.8/2.5 at 16.8 MB, at 8.4 MB no gain, so the line lies
// between.  With 4 of the cores 14.8/4.9 at 33.6 MB; with one the first copy
// lost (6.7/7.5).  Copies to the device go the driver's way: 33.6 MB took the
// threads 2.4, the driver 1.8 from a source in the CPU's caches and 3.2 else.
constexpr size_t kStagedFrom = 16 << 20;
constexpr int kMinCpus = 4;
constexpr size_t kPiece = 128 << 10;  // larger pieces pin more: the first copy was slower than the driver's from 512 KB on
constexpr int kThreads = 6;

// one thread's buffers and stream
struct Lane {
    void* buf[2] = {nullptr, nullptr};
    cudaStream_t stream = nullptr;
    cudaEvent_t landed[2] = {nullptr, nullptr};
};
struct Staging {
    Lane lanes[kThreads];
    char* pinned = nullptr;  // the lanes' buffers, one allocation
    bool ok = false;
};

void host_copy_free(bdc_handle* H) {
    Staging* S = (Staging*)H->staging;
    H->staging = nullptr;
    if (!S) return;
    for (Lane& l : S->lanes) {
        for (int i = 0; i < 2; ++i) {
            if (l.landed[i]) cudaEventDestroy(l.landed[i]);
        }
        if (l.stream) cudaStreamDestroy(l.stream);
    }
    if (S->pinned) cudaFreeHost(S->pinned);
    delete S;
}

// the handle's buffers (1.5 MB pinned), or null when they cannot be had
static Staging* staging(bdc_handle* H) {
    Staging* S = (Staging*)H->staging;
    if (S) return S->ok ? S : nullptr;
    S = new (std::nothrow) Staging();
    if (!S) return nullptr;
    H->staging = S;
    cudaError_t e = cudaMallocHost(&S->pinned, 2 * kThreads * kPiece);
    char* at = S->pinned;
    for (Lane& l : S->lanes) {
        for (int i = 0; i < 2 && e == cudaSuccess; ++i, at += kPiece) {
            l.buf[i] = at;
            e = cudaEventCreateWithFlags(&l.landed[i], cudaEventDisableTiming);
        }
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking);
    }
    S->ok = e == cudaSuccess;
    if (!S->ok) (void)cudaGetLastError();  // the plain copy serves
    return S->ok ? S : nullptr;
}

// most of the pages of [p, p + bytes) have no memory behind them yet, by a
// sample of them (16 us for 64 pages)
static bool fresh_pages(const void* p, size_t bytes) {
    constexpr int kSample = 64;
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    int fresh = 0;
    for (int i = 0; i < kSample; ++i) {
        unsigned char in = 1;
        const uintptr_t at = ((uintptr_t)p + bytes / kSample * i) / page * page;
        if (mincore((void*)at, page, &in) != 0) return false;
        fresh += !(in & 1);
    }
    return fresh > kSample / 2;
}

static bool enough_cpus() {
    cpu_set_t set;
    CPU_ZERO(&set);
    return sched_getaffinity(0, sizeof(set), &set) == 0 && CPU_COUNT(&set) >= kMinCpus;
}

// every kThreads-th piece from piece t on; returns with its copies complete
static cudaError_t run_lane(int device, Lane& l, int t, char* dst, const char* src, size_t bytes) {
    cudaError_t e = cudaSetDevice(device);
    const size_t stride = kPiece * kThreads;
    auto queue = [&](int i, size_t at) {
        const cudaError_t c =
            cudaMemcpyAsync(l.buf[i], src + at, std::min(kPiece, bytes - at), cudaMemcpyDeviceToHost, l.stream);
        return c != cudaSuccess ? c : cudaEventRecord(l.landed[i], l.stream);
    };
    int i = 0;
    size_t at = kPiece * (size_t)t;
    if (e == cudaSuccess && at < bytes) e = queue(i, at);
    for (; at < bytes && e == cudaSuccess; at += stride, i ^= 1) {
        if (at + stride < bytes) e = queue(i ^ 1, at + stride);
        if (e == cudaSuccess) e = cudaEventSynchronize(l.landed[i]);
        if (e == cudaSuccess) memcpy(dst + at, l.buf[i], std::min(kPiece, bytes - at));
    }
    const cudaError_t e2 = cudaStreamSynchronize(l.stream);
    return e != cudaSuccess ? e : e2;
}

cudaError_t copy_to_host(bdc_handle* H, void* dst, const void* src, size_t bytes) {
    Staging* S = nullptr;
    if (bytes >= kStagedFrom) {
        cudaPointerAttributes at{};
        if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) (void)cudaGetLastError();
        if (at.type == cudaMemoryTypeUnregistered && enough_cpus() && fresh_pages(dst, bytes)) S = staging(H);
    }
    if (!S) {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, H->stream);
        return e != cudaSuccess ? e : cudaStreamSynchronize(H->stream);
    }
    // the lanes' streams do not follow H->stream: it must be idle
    cudaError_t e = cudaStreamSynchronize(H->stream);
    if (e != cudaSuccess) return e;
    std::thread threads[kThreads];
    cudaError_t got[kThreads] = {};
    int started = 0;
    try {
        for (; started + 1 < kThreads; ++started) {
            const int t = started + 1;
            threads[t] = std::thread([=, &got] {
                got[t] = run_lane(H->device, S->lanes[t], t, (char*)dst, (const char*)src, bytes);
            });
        }
    } catch (const std::exception&) {  // no more threads: this one takes the rest
    }
    got[0] = run_lane(H->device, S->lanes[0], 0, (char*)dst, (const char*)src, bytes);
    for (int t = started + 1; t < kThreads; ++t)
        got[t] = run_lane(H->device, S->lanes[t], t, (char*)dst, (const char*)src, bytes);
    for (int t = 1; t <= started; ++t) threads[t].join();
    for (cudaError_t g : got)
        if (g != cudaSuccess) return g;
    return cudaSuccess;
}

}  // namespace bdc
