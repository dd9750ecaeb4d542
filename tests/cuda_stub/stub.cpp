// A stand-in for the CUDA runtime and the kernel launchers, so that the host
// side of the C ABI (rtdbs_engine.cpp) runs on a machine without a GPU: every
// call is counted by name, memory comes from malloc, copies and sets are done
// when called, launches only record what they were given.  Memory registered
// with stub_memory has the kind and the extent that the engine then sees.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

#include "rtdbs.h"
#include "rtdbs_internal.h"

namespace {

struct Range {
    size_t bytes;
    cudaMemoryType type;
};
std::map<uintptr_t, Range> g_memory;  // by first byte
std::map<std::string, int> g_calls;
size_t g_pinned_limit = ~size_t(0);   // largest cudaMallocHost that succeeds
rtdbs::SlideIO g_io;                  // of the last first kernel of a slide or load
int g_runs = 0;                       // cell runs and distance tests that a whole
unsigned long long g_tests = 0;       // build reports
int g_lanes = 0;                      // lanes per query of the last launch
int g_warps = 5472;                   // count_pass_warps()

cudaError_t count(const char* name) {
    ++g_calls[name];
    return cudaSuccess;
}

void* take(size_t bytes, cudaMemoryType type) {
    void* p = std::calloc(bytes ? bytes : 1, 1);
    g_memory[(uintptr_t)p] = {bytes, type};
    return p;
}

const Range* find(const void* p, uintptr_t* base) {
    auto it = g_memory.upper_bound((uintptr_t)p);
    if (it == g_memory.begin()) return nullptr;
    --it;
    if ((uintptr_t)p >= it->first + it->second.bytes) return nullptr;
    *base = it->first;
    return &it->second;
}

// Whether `bytes` from p on lie within one known allocation (plain host
// memory is not known, and passes).
bool inside(const void* p, size_t bytes) {
    uintptr_t base = 0;
    const Range* r = find(p, &base);
    return !r || (uintptr_t)p + bytes <= base + r->bytes;
}

int address_range(unsigned long long* base, size_t* bytes, unsigned long long p) {
    uintptr_t b = 0;
    const Range* r = find((const void*)p, &b);
    count("cuMemGetAddressRange");
    if (!r || r->type != cudaMemoryTypeDevice) return 1;
    *base = b;
    *bytes = r->bytes;
    return 0;
}

}  // namespace

extern "C" {

int stub_calls(const char* name) { return g_calls[name]; }
void stub_reset() { g_calls.clear(); }
void stub_pinned_limit(size_t bytes) { g_pinned_limit = bytes; }
void stub_warps(int n) { g_warps = n; }
void stub_window(int runs, unsigned long long tests) { g_runs = runs; g_tests = tests; }
int stub_lanes() { return g_lanes; }
void* stub_memory(size_t bytes, int type) { return take(bytes, (cudaMemoryType)type); }
const void* stub_io(int which) { return which == 0 ? g_io.input : which == 1 ? (void*)g_io.label : (void*)g_io.cid; }

// Cells of n coordinates on axis 0 of the grid over [lo, hi]; also the grid's
// extent there, its cell side and the largest error that the single-precision
// quotient is trusted with.
int stub_cells(double eps, int cells, float lo, float hi, const float* x, long long n, long long* cell,
               long long* extent, double* side, float* key_err) {
    rtdbs::View v{};
    const int rc = rtdbs::set_geometry(v, 1, eps, cells, &lo, &hi, false, side);
    if (rc != RTDBS_OK) return rc;
    for (long long i = 0; i < n; ++i) cell[i] = rtdbs::cell_coord(v, 0, x[i]);
    *extent = v.ext[0];
    *key_err = v.key_err[0];
    return RTDBS_OK;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stub"; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = take(n, cudaMemoryTypeDevice); return count("cudaMalloc"); }
cudaError_t cudaMallocHost(void** p, size_t n) {
    if (n > g_pinned_limit) return cudaErrorMemoryAllocation;
    *p = take(n, cudaMemoryTypeHost);
    return count("cudaMallocHost");
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) { g_memory.erase((uintptr_t)p); std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (!inside(d, n) || !inside(s, n)) return cudaErrorInvalidValue;
    std::memmove(d, s, n);
    return count("cudaMemcpyAsync");
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, 0); }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaStreamCreate(cudaStream_t* s) { return cudaStreamCreateWithFlags(s, 0); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)std::malloc(16);
    return count("cudaStreamCreate");
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free((void*)s); return count("cudaStreamDestroy"); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return count("cudaStreamSynchronize"); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return count("cudaStreamWaitEvent"); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = (cudaEvent_t)std::malloc(16);
    return count("cudaEventCreate");
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free((void*)e); return count("cudaEventDestroy"); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return count("cudaEventRecord"); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)std::malloc(16); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    *x = (cudaGraphExec_t)std::malloc(16);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { std::free((void*)g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { std::free((void*)x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return count("cudaGraphLaunch"); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    uintptr_t base = 0;
    const Range* r = find(p, &base);
    std::memset(a, 0, sizeof(*a));
    a->type = r ? r->type : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
    const bool known = std::strcmp(name, "cuMemGetAddressRange") == 0;
    *f = known ? (void*)address_range : nullptr;
    if (r) *r = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}

}  // extern "C"

namespace rtdbs {

cudaError_t launch_phase(int phase, const View&, int, int j, int, int, int, int, cudaStream_t, bool, const SlideIO& io) {
    if (phase == kPhaseIngest && j == 0) g_io = io;
    return count("launch");
}
cudaError_t launch_chunk_step(const View&, int, int, int, int, int, cudaStream_t, const SlideIO& io, bool ingested,
                              cudaStream_t, cudaEvent_t, cudaEvent_t) {
    if (!ingested && io.input) g_io = io;
    return count("launch");
}
cudaError_t launch_window_build(const View& v, int, const SlideIO& io, int, int, cudaStream_t, bool ingested) {
    g_lanes = v.qlanes;
    if (!ingested) g_io = io;
    v.ctl->nitems = g_runs;
    v.ctl->ptests[0][0] = g_tests;
    count("launch_window_build");
    return count("launch");
}
cudaError_t launch_window_phase(int phase, const View&, int, const SlideIO& io, int, int, cudaStream_t, bool) {
    if (phase == kPhaseIngest) g_io = io;
    return count("launch");
}
int window_build_launches(const View&) { return 5; }
cudaError_t launch_bbox(const float*, long long, int, unsigned* box, cudaStream_t) {
    for (int a = 0; a < 6; ++a) box[a] = a < 3 ? 0x80000000u : 0xc2c80000u;  // 0 to 100
    return count("launch_bbox");
}
cudaError_t launch_cluster(const View&, int, int, cudaStream_t, bool, cudaEvent_t, unsigned, const SlideIO& io) {
    if (io.label || io.cid) g_io = io;
    return count("launch");
}
cudaError_t launch_counts_by_slot(const View&, int*, cudaStream_t) { return count("launch"); }
cudaError_t configure_kernels() { return cudaSuccess; }
int count_pass_warps() { return g_warps; }
int batch_blocks(int, const View&, int) { return 1; }
int batch_threads(int) { return 256; }
bool batch_phase_split(int) { return false; }
cudaError_t launch_batch(int, int, int, const BatchLaunch&, int, int, cudaStream_t) { return count("launch_batch"); }
cudaError_t launch_gather(const float* const*, const long long*, const int*, float*, int, int, cudaStream_t) {
    return count("launch_gather");
}

}  // namespace rtdbs
