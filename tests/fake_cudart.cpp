// A CUDA runtime without a device, preloaded over libcudart so that the host
// code of libbdc_b200.so runs where there is no GPU: device memory is host
// memory, copies happen at once, kernels do nothing (the list of
// representatives is written for them, and an iteration's last kernel counts).  What the runtime or the device would
// only show now and then is checked on each call instead: copies out of an
// allocation's range, a copy on the legacy stream over work that a
// non-blocking stream still has queued, products outside their operands and
// results, launches without blocks or with more
// shared memory than the kernel's limit.  A test can let allocations fail and
// let a kernel leave an error code in the device state.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

#define __ldg(p) (*(p))
#include <cmath>
using std::isfinite;
#include "../bdc-upper-bounds-gpu_b200/csrc/bdc_gemm.cuh"

namespace {

struct Block {
    size_t bytes;
    bool device, written;
};
struct Pending {
    cudaStream_t s;
    const char* at;
    size_t bytes;
    uint64_t seq;
};
struct Copy {
    int kind;
    size_t bytes;
};
struct World {
    std::recursive_mutex mu;
    std::map<const char*, Block> blocks;
    std::vector<Pending> pending;   // queued writes of non-blocking streams
    std::map<cudaEvent_t, std::pair<cudaStream_t, uint64_t>> events;
    std::map<const void*, std::string> kernels;
    std::map<const void*, int> smem_limit;
    std::map<const void*, std::pair<char*, size_t>> vars;
    std::map<std::string, long> launches, grids;
    std::map<void*, int> graphs;  // iterations that a captured graph holds
    int iterations = 0;           // of the capture that is open or was last
    std::vector<Copy> copies;
    std::string faults;
    cudaStream_t capturing = nullptr;
    uint64_t seq = 0;
    uintptr_t next = 0x1000;
    size_t fail_from = SIZE_MAX;
    std::string fault_kernel;
    int fault_code = 0;
    long long stop_after = INT64_MAX;  // the iteration that meets the threshold
    std::vector<uint32_t> reps;
    cudaError_t last = cudaSuccess;
};
World& W() {
    static World* w = new World();
    return *w;
}
using Lock = std::lock_guard<std::recursive_mutex>;

void fault(const char* what, const std::string& where = "") { W().faults += std::string(what) + " " + where + "\n"; }

// the block that holds p, or end
std::map<const char*, Block>::iterator find(const void* p) {
    auto& b = W().blocks;
    auto it = b.upper_bound((const char*)p);
    if (it == b.begin()) return b.end();
    --it;
    return (const char*)p < it->first + it->second.bytes ? it : b.end();
}
void in_range(const void* p, size_t bytes, const char* what) {
    auto it = find(p);
    if (it != W().blocks.end() && (const char*)p + bytes > it->first + it->second.bytes) fault("out of range:", what);
}
void settle(cudaStream_t s, uint64_t upto) {
    auto& v = W().pending;
    std::vector<Pending> keep;
    for (auto& q : v)
        if (!(q.s == s && q.seq <= upto)) keep.push_back(q);
    v.swap(keep);
}
bool captured(cudaStream_t s) { return W().capturing && s == W().capturing; }

cudaError_t transfer(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t s, bool legacy) {
    Lock l(W().mu);
    if (!legacy && W().capturing) return cudaSuccess;  // a node of the graph
    in_range(dst, bytes, "copy destination");
    in_range(src, bytes, "copy source");
    if (legacy)
        for (auto& q : W().pending)
            if (q.at < (const char*)dst + bytes && (const char*)dst < q.at + q.bytes)
                fault("unordered: a copy over a range that a non-blocking stream has still to write");
    if (!legacy && s && kind == cudaMemcpyHostToDevice)
        W().pending.push_back({s, (const char*)dst, bytes, ++W().seq});
    auto it = find(dst);
    if (it != W().blocks.end()) it->second.written = true;
    if (bytes) memmove(dst, src, bytes);
    W().copies.push_back({(int)kind, bytes});
    return cudaSuccess;
}

bool named(const std::string& mangled, const char* name) {
    return mangled.find(std::to_string(strlen(name)) + name) != std::string::npos;
}

void advance(int iterations) {
    for (auto& b : W().blocks)
        if (b.second.device && b.second.bytes == sizeof(bdc::DevState)) {
            auto* st = (bdc::DevState*)b.first;
            for (int i = 0; i < iterations && !st->done; ++i) st->done = ++st->iter >= W().stop_after;
            b.second.written = true;
        }
}

// what the tiles of a grouped product read and write
void check_products(const bdc::GemmDesc* d, const int* map, unsigned tiles) {
    in_range(map, sizeof(int) * tiles, "tile map");
    for (unsigned t = 0; t < tiles; ++t) {
        if (t > 0 && map[t] == map[t - 1]) continue;
        const bdc::GemmDesc& e = d[map[t]];
        in_range(&e, sizeof(e), "product descriptor");
        auto operand = [&](const bdc::Operand& o, int64_t rows, int64_t cols, const char* what) {
            if (rows < 1 || cols < 1) return;
            const int64_t end = (o.trans ? (cols - 1) * o.ld + rows : (rows - 1) * o.ld + cols);
            if (find(o.ptr) == W().blocks.end()) fault("out of range:", what);
            in_range(o.ptr, 8 * end, what);
        };
        operand(e.A, e.M, e.K, "product operand A");
        operand(e.B, e.K, e.N, "product operand B");
        const int64_t end = (e.M - 1) * e.ldc_m + (e.N - 1) * e.ldc_n + 1;
        if (e.K < 0 || find(e.C) == W().blocks.end()) fault("out of range:", "product result");
        in_range(e.C, 8 * end, "product result");
    }
}

cudaError_t launch(const void* f, dim3 grid, void** args, size_t smem) {
    World& w = W();
    Lock l(w.mu);
    const std::string& name = w.kernels[f];
    const int limit = w.smem_limit.count(f) ? w.smem_limit[f] : 48 * 1024;
    if (grid.x == 0 || smem > (size_t)limit) {
        fault(grid.x == 0 ? "launch of no blocks:" : "launch above the shared memory limit:", name);
        return w.last = cudaErrorInvalidValue;
    }
    w.launches[name] += 1;
    w.grids[name] = grid.x;
    if (named(name, "k_mma_store")) check_products(*(const bdc::GemmDesc**)args[0], *(const int**)args[1], grid.x);
    // the iterations that this launch ends: k_direct does what & 2 of one, or `iters` alone
    int done = named(name, "k_fac_finalize");
    if (named(name, "k_direct") && (*(int*)args[1] & 2)) done = name.find("Lb1E") != name.npos ? *(int*)args[3] : 1;
    if (w.capturing) {
        w.iterations += done;
        return cudaSuccess;
    }
    if (done) advance(done);
    if (named(name, "k_rep_count")) {
        const int n = *(int*)args[0];
        w.reps.clear();
        for (uint32_t x = 0; x < (1u << (n - 1)); ++x) {  // a representative's top bit is 0
            uint32_t r = __builtin_bswap32(x);
            r = (r & 0x0F0F0F0Fu) << 4 | (r >> 4 & 0x0F0F0F0Fu);
            r = (r & 0x33333333u) << 2 | (r >> 2 & 0x33333333u);
            r = ((r & 0x55555555u) << 1 | (r >> 1 & 0x55555555u)) >> (32 - n);
            if (x <= r && x <= (r ^ bdc::low_mask(n))) w.reps.push_back(x);
        }
    } else if (named(name, "k_rep_scan")) {
        **(int64_t**)args[2] = (int64_t)w.reps.size();
    } else if (named(name, "k_rep_write")) {
        uint32_t* to = *(uint32_t**)args[2];
        memcpy(to, w.reps.data(), 4 * w.reps.size());
        find(to)->second.written = true;
    } else if (!w.fault_kernel.empty() && name.find(w.fault_kernel) != std::string::npos) {
        for (auto& b : w.blocks)
            if (b.second.device && b.second.bytes == sizeof(bdc::DevState))
                ((bdc::DevState*)b.first)->error = w.fault_code;
    }
    return cudaSuccess;
}

struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t s;
};
thread_local std::vector<Config> t_config;

int encode_tiled() { return 0; }

}  // namespace

extern "C" {

// ---- what a test reads and sets
const char* fake_faults() { return W().faults.c_str(); }
void fake_clear() {
    Lock l(W().mu);
    W().faults.clear();
    W().copies.clear();
    W().launches.clear();
}
void fake_fail_malloc(size_t from_bytes) { W().fail_from = from_bytes; }
void fake_fault_in(const char* kernel, int code) {
    Lock l(W().mu);
    W().fault_kernel = kernel;
    W().fault_code = code;
}
void fake_stop_after(int iterations) { W().stop_after = iterations; }
long fake_launches(const char* part) {
    Lock l(W().mu);
    long t = 0;
    for (auto& kv : W().launches)
        if (kv.first.find(part) != std::string::npos) t += kv.second;
    return t;
}
long fake_grid(const char* kernel) {  // blocks of the kernel's last launch
    Lock l(W().mu);
    for (auto& kv : W().grids)
        if (named(kv.first, kernel)) return kv.second;
    return 0;
}
long fake_copies(int kind, size_t from_bytes) {
    Lock l(W().mu);
    long t = 0;
    for (auto& c : W().copies) t += c.kind == kind && c.bytes >= from_bytes;
    return t;
}

// ---- memory
static cudaError_t get(void** p, size_t bytes, bool device) {
    Lock l(W().mu);
    *p = nullptr;
    if (bytes >= W().fail_from) return W().last = cudaErrorMemoryAllocation;
    *p = calloc(1, bytes + 256);
    if (!*p) return W().last = cudaErrorMemoryAllocation;
    W().blocks[(const char*)*p] = Block{bytes, device, false};
    return cudaSuccess;
}
static cudaError_t put(void* p) {
    Lock l(W().mu);
    if (!p) return cudaSuccess;
    W().blocks.erase((const char*)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes) { return get(p, bytes, true); }
cudaError_t cudaFree(void* p) { return put(p); }
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { return get(p, bytes, false); }
cudaError_t cudaMallocHost(void** p, size_t bytes) { return get(p, bytes, false); }
cudaError_t cudaFreeHost(void* p) { return put(p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    *f = *t = (size_t)180 << 30;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
    return transfer(dst, src, bytes, kind, nullptr, true);
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t s) {
    return transfer(dst, src, bytes, kind, s, false);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t s) {
    Lock l(W().mu);
    if (W().capturing) return cudaSuccess;
    in_range(p, bytes, "memset");
    auto it = find(p);
    if (it != W().blocks.end() && (v != 0 || it->second.written)) memset(p, v, bytes);
    if (s) W().pending.push_back({s, (const char*)p, bytes, ++W().seq});
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    Lock l(W().mu);
    memset(a, 0, sizeof(*a));
    auto it = find(p);
    a->type = it == W().blocks.end() ? cudaMemoryTypeUnregistered
                                     : it->second.device ? cudaMemoryTypeDevice : cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) {
    *p = W().vars[sym].first;
    return *p ? cudaSuccess : cudaErrorInvalidSymbol;
}

// ---- streams, events, graphs
static void* handle() {
    Lock l(W().mu);
    return (void*)(W().next += 16);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)handle();
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    Lock l(W().mu);
    settle(s, UINT64_MAX);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t)handle();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    Lock l(W().mu);
    W().events[e] = {s, W().seq};
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    Lock l(W().mu);
    auto it = W().events.find(e);
    if (it != W().events.end()) settle(it->second.first, it->second.second);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 5.f;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    W().capturing = s;
    W().iterations = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    W().capturing = nullptr;
    *g = (cudaGraph_t)handle();
    W().graphs[*g] = W().iterations;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    *e = (cudaGraphExec_t)handle();
    W().graphs[*e] = W().graphs[g];
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    Lock l(W().mu);
    advance(W().graphs[e]);
    return cudaSuccess;
}

// ---- device
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 1;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = W().last;
    W().last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* r) {
    *f = (void*)&encode_tiled;
    if (r) *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

// ---- kernels
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    Lock l(W().mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) W().smem_limit[f] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void** args, size_t smem, cudaStream_t) {
    return launch(f, grid, args, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return launch(f, c->gridDim, args, c->dynamicSmemBytes);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    t_config.push_back({grid, block, smem, s});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
    const Config c = t_config.back();
    t_config.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *(cudaStream_t*)s = c.s;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
    static void* one = nullptr;
    return &one;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    Lock l(W().mu);
    W().kernels[host] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t bytes, int, int) {
    Lock l(W().mu);
    W().vars[host] = {(char*)calloc(1, bytes + 16), bytes};
}

}  // extern "C"
