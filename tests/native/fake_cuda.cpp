/*
 * fake_cuda.cpp -- test-only stand-in for the CUDA runtime and the kernel
 * launchers under the library's host sources (lbm_host.cpp, lbm_sgs.cpp,
 * lbm_ensemble.cpp), so that their bookkeeping and their error paths run
 * without a GPU: device memory is host memory, work on a stream is done at
 * once, kernels do nothing.  Every other symbol that the sources need is a
 * function that returns 0 (conftest.py generates them).  Not part of the
 * product library.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>
#include <sys/mman.h>

#include <algorithm>
#include <map>
#include <string>
#include <vector>

#include "../../lbm_multigpu_gb300/csrc/lbm_kernels.cuh"
#include "../../lbm_multigpu_gb300/csrc/sgs_infer.cuh"

namespace {
std::map<void*, size_t> g_mem;
std::map<std::string, long> g_calls, g_fail_at;
std::map<std::string, size_t> g_fail_above;
std::vector<long long> g_trace;
int g_device = 0;
std::vector<uint8_t> g_mask;                   /* of the last step */
std::vector<uint32_t> g_links, g_body, g_blinks; /* and of the last force */
const int* g_perm = nullptr; /* the permutation that a shuffle last filled */

/* counts the call; true when a test asked for it to fail */
bool failing(const char* fn, size_t bytes = 0) {
    const long n = ++g_calls[fn];
    if (g_fail_at.count(fn) && g_fail_at[fn] == n) return true;
    return g_fail_above.count(fn) && bytes > g_fail_above[fn];
}
cudaError_t take(void** p, size_t n) {
    /* address space only: a test may ask for more than the machine has */
    void* m = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
    g_mem[m] = n ? n : 1;
    *p = m;
    return cudaSuccess;
}
cudaError_t give(void* p) {
    if (!p) return cudaSuccess;
    if (!g_mem.count(p)) return cudaErrorInvalidValue;
    munmap(p, g_mem[p]);
    g_mem.erase(p);
    return cudaSuccess;
}
}  // namespace

extern "C" {

/* for the tests: the call number `at` of fn from now on fails (0: none), or every one for more than `bytes` bytes */
void fake_fail(const char* fn, long at) { g_fail_at[fn] = at ? g_calls[fn] + at : 0; }
void fake_fail_above(const char* fn, size_t bytes) { g_fail_above[fn] = bytes; }
long fake_calls(const char* fn) { return g_calls[fn]; }
size_t fake_blocks() { return g_mem.size(); }
/* what the launchers below noted */
long fake_trace(long long* out, long cap) {
    const long n = long(g_trace.size());
    for (long i = 0; i < n && i < cap; ++i) out[i] = g_trace[i];
    return n;
}
long fake_mask(uint8_t* out) { return std::copy(g_mask.begin(), g_mask.end(), out) - out; }
long fake_words(int which, uint32_t* out, long cap) {
    const std::vector<uint32_t>& v = which == 0 ? g_links : which == 1 ? g_body : g_blinks;
    for (long i = 0; i < cap && i < long(v.size()); ++i) out[i] = v[i];
    return long(v.size());
}
void fake_reset() {
    g_body.clear(), g_blinks.clear();
    g_calls.clear(), g_fail_at.clear(), g_fail_above.clear(), g_trace.clear(), g_perm = nullptr;
}

/* the grid of one kernel on a device: 100 (device + 1), or an error when `fails` */
int fake_device_grid(int device, int fails, int* grid) {
    static lbm::sgs::DeviceGrids grids;
    g_device = device;
    const cudaError_t e = grids.get(
        [&](int* g) {
            ++g_calls["grid"];
            *g = 100 * (device + 1);
            return fails ? cudaErrorUnknown : cudaSuccess;
        },
        grid);
    g_device = 0;
    return int(e);
}

cudaError_t cudaMalloc(void** p, size_t n) { return failing("cudaMalloc", n) ? cudaErrorMemoryAllocation : take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    return failing("cudaMallocFromPoolAsync", n) ? cudaErrorMemoryAllocation : take(p, n);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (failing("cudaMemcpy", n)) return cudaErrorUnknown;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (failing("cudaMemcpyAsync", n)) return cudaErrorUnknown;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    if (failing("cudaMemcpy2DAsync", w * h)) return cudaErrorUnknown;
    for (size_t i = 0; i < h; ++i) memcpy(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = g_device, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) { return *a = *b = 0, cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    return *a = cudaPointerAttributes{}, cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
/* handles are numbers; of a step graph's executable the stand-in keeps when it was last built or updated */
static uintptr_t g_next = 0;
static std::map<cudaGraphExec_t, uintptr_t> g_built;
static uintptr_t g_mark = 0;
static long g_stale = 0;
/* from here on: the launches of executables last built before this call */
void fake_mark() { g_mark = ++g_next, g_stale = 0; }
long fake_stale_launches() { return g_stale; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    return failing("cudaStreamBeginCapture") ? cudaErrorIllegalState : cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = reinterpret_cast<cudaGraph_t>(++g_next);
    return failing("cudaStreamEndCapture") ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    if (failing("cudaGraphInstantiate")) return cudaErrorUnknown;
    *x = reinterpret_cast<cudaGraphExec_t>(++g_next);
    g_built[*x] = g_next;
    return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t x, cudaGraph_t, cudaGraphExecUpdateResultInfo*) {
    if (failing("cudaGraphExecUpdate")) return cudaErrorUnknown;
    g_built[x] = ++g_next;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    if (failing("cudaGraphLaunch")) return cudaErrorUnknown;
    g_stale += g_built[x] < g_mark;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(++g_next), cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    return *e = reinterpret_cast<cudaEvent_t>(++g_next), cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    return *p = reinterpret_cast<cudaMemPool_t>(++g_next), cudaSuccess;
}

}  // extern "C"

namespace lbm {
int force_partials() { return 608; }
cudaError_t launch_force(const Level&, const void*, const unsigned* body, int nbody, double*, unsigned*, double*, cudaStream_t,
                         const uint32_t* blinks, const int*) {
    g_calls["launch_force"]++;
    if (nbody <= 0) return cudaSuccess;
    if (!body) return g_calls["null body list"]++, cudaErrorInvalidValue;
    g_body.assign(body, body + nbody);
    g_blinks.assign(blinks, blinks ? blinks + nbody : blinks);
    return cudaSuccess;
}
/* every word of the statistics is its own index (below 2^24) */
cudaError_t launch_stream_collide(const Level& L, const StepParams&, const void*, void*, const uint8_t* mask, float* stats,
                                  float*, cudaStream_t, const uint32_t* links) {
    g_mask.assign(mask, mask + L.qstride);
    g_links.assign(links, links ? links + L.qstride : links);
    for (long long i = 0; stats && i < 4 * L.qstride; ++i) stats[i] = float(i);
    return cudaSuccess;
}
int ens_step_resident(int, int) { return 608; }
int mlp_grad_blocks(int) { return 1; }
size_t shuffle_scratch_bytes(int n) { return 20 * size_t(n); }
cudaError_t launch_shuffle(int* perm, int, unsigned long long, int, void*, cudaStream_t) {
    g_calls["launch_shuffle"]++;
    g_perm = perm;
    return cudaSuccess;
}
/* notes where the batch begins and its size; after an upload of the sample order, its elements instead */
cudaError_t launch_mlp_grad(const float*, const float*, const float*, const int* idx, int n, float*, int, cudaStream_t) {
    if (!g_perm && g_calls["cudaMemcpyAsync"] > 1) { /* one upload is the parameters' */
        g_trace.insert(g_trace.end(), idx, idx + n);
        return cudaSuccess;
    }
    g_trace.push_back(g_perm ? idx - g_perm : -1); /* -1: nothing filled the permutation yet */
    g_trace.push_back(n);
    return cudaSuccess;
}
}  // namespace lbm
