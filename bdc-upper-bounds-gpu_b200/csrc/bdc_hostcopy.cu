// bdc_hostcopy.cu -- vectors of representatives between pageable host memory
// and the device.
//
// The driver copies pageable memory through one pinned buffer on the calling
// thread: 33.6 MB (24/12) took 1.8 ms in and 6.8 ms out, the latter mostly the
// first touch of the caller's fresh pages.  Here a few threads each take every
// kThreads-th piece of 128 KB through two pinned buffers of their own, one being
// filled by the DMA engine while the other is copied, so that the copies and
// the page faults run in parallel.  Small and pinned copies go as before.
#include <algorithm>
#include <cstring>
#include <exception>
#include <new>
#include <thread>

#include "bdc_engine.cuh"

namespace bdc {

// A host-vector iteration at 24/12 (two copies of 33.6 MB), a handle's first,
// which pins the buffers, and later ones: 10.7-11.1 ms through the driver; pieces
// of 1 MB 10-17 and 3.1, 512 KB 8-14 and 3.8, 256 KB 8.4-11.4 and 4.6, 128 KB 6-9 and 5.5.
// (the largest that leaves the first call no slower than the driver's copies)
constexpr size_t kPiece = 128 << 10;
constexpr size_t kStagedFrom = 4 << 20;  // below this the threads cost what they give (0.46 against 0.41 ms a step at 2.1 MB)
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

// every kThreads-th piece from piece t on; returns with its copies complete
static cudaError_t run_lane(int device, Lane& l, int t, char* dst, const char* src, size_t bytes, bool to_host) {
    cudaError_t e = cudaSetDevice(device);
    const size_t stride = kPiece * kThreads;
    auto size = [&](size_t at) { return std::min(kPiece, bytes - at); };
    int i = 0;
    bool ahead = false;  // (to the host) the current piece's copy is already queued
    for (size_t at = kPiece * (size_t)t; at < bytes && e == cudaSuccess; at += stride, i ^= 1) {
        if (to_host) {
            if (!ahead) {
                e = cudaMemcpyAsync(l.buf[i], src + at, size(at), cudaMemcpyDeviceToHost, l.stream);
                if (e == cudaSuccess) e = cudaEventRecord(l.landed[i], l.stream);
            }
            const size_t next = at + stride;
            ahead = next < bytes;
            if (e == cudaSuccess && ahead) {
                e = cudaMemcpyAsync(l.buf[i ^ 1], src + next, size(next), cudaMemcpyDeviceToHost, l.stream);
                if (e == cudaSuccess) e = cudaEventRecord(l.landed[i ^ 1], l.stream);
            }
            if (e == cudaSuccess) e = cudaEventSynchronize(l.landed[i]);
            if (e == cudaSuccess) memcpy(dst + at, l.buf[i], size(at));
        } else {
            e = cudaEventSynchronize(l.landed[i]);  // the buffer's last copy is done
            if (e != cudaSuccess) break;
            memcpy(l.buf[i], src + at, size(at));
            e = cudaMemcpyAsync(dst + at, l.buf[i], size(at), cudaMemcpyHostToDevice, l.stream);
            if (e == cudaSuccess) e = cudaEventRecord(l.landed[i], l.stream);
        }
    }
    const cudaError_t e2 = cudaStreamSynchronize(l.stream);
    return e != cudaSuccess ? e : e2;
}

cudaError_t host_copy(bdc_handle* H, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
    const bool to_host = kind == cudaMemcpyDeviceToHost;
    Staging* S = nullptr;
    if (bytes >= kStagedFrom) {
        cudaPointerAttributes at{};
        if (cudaPointerGetAttributes(&at, to_host ? dst : src) != cudaSuccess) (void)cudaGetLastError();
        if (at.type == cudaMemoryTypeUnregistered) S = staging(H);
    }
    if (!S) {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, kind, H->stream);
        return e != cudaSuccess || !to_host ? e : cudaStreamSynchronize(H->stream);
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
                got[t] = run_lane(H->device, S->lanes[t], t, (char*)dst, (const char*)src, bytes, to_host);
            });
        }
    } catch (const std::exception&) {  // no more threads: this one takes the rest
    }
    got[0] = run_lane(H->device, S->lanes[0], 0, (char*)dst, (const char*)src, bytes, to_host);
    for (int t = started + 1; t < kThreads; ++t)
        got[t] = run_lane(H->device, S->lanes[t], t, (char*)dst, (const char*)src, bytes, to_host);
    for (int t = 1; t <= started; ++t) threads[t].join();
    for (cudaError_t g : got)
        if (g != cudaSuccess) return g;
    return cudaSuccess;
}

}  // namespace bdc
