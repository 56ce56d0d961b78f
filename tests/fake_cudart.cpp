// A stand-in for the CUDA runtime, for tests of the library's host side on a
// machine without a GPU (test_host_runtime.py loads it in the runtime's place).
// Device memory is host memory and kernels do nothing; what is modelled is what
// the host code must get right:
//   * function attributes belong to the device current when they are set, and a
//     launch that asks for more dynamic shared memory than the device's limit
//     for that kernel (48 KiB unless raised) is refused;
//   * the order of operations: every launch, copy, event record and wait goes to
//     a log with its stream.
// Two devices.  fake_set("clusters", 0) makes clusters unlaunchable by the
// occupancy query, fake_set("refuse_clusters", 1) their launches alone,
// fake_set("pinned_failures", n) fails the next n pinned allocations,
// fake_set("malloc_failure_at", n) the n-th device allocation from then on.
#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

namespace {

std::recursive_mutex m;
int g_dev = 0, g_clusters = 8, g_pinned_failures = 0, g_malloc_failure_at = 0, g_refuse_clusters = 0;
cudaError_t g_last = cudaSuccess;
std::map<const void*, std::string> g_names;
std::map<const void*, size_t> g_vars;
std::map<std::pair<int, const void*>, size_t> g_limit;
std::map<std::pair<int, const void*>, void*> g_symbols;
std::map<cudaStream_t, unsigned long long> g_stream_ids;
std::map<cudaStream_t, bool> g_capturing;
std::vector<std::string> g_log;
unsigned long long g_next = 1;

struct Call { dim3 grid, block; size_t smem; cudaStream_t st; };
std::vector<Call> g_calls;

cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}
void log_op(const char* f, ...) {
    char b[512];
    va_list a;
    va_start(a, f);
    vsnprintf(b, sizeof(b), f, a);
    va_end(a);
    g_log.push_back(b);
}
template <class H>
H handle() {
    return (H)(uintptr_t)(0x10000 + 16 * g_next++);
}
cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    const auto it = g_limit.find({g_dev, f});
    const size_t limit = it == g_limit.end() ? 48 * 1024 : it->second;
    const auto n = g_names.find(f);
    const char* name = n == g_names.end() ? "?" : n->second.c_str();
    if (smem > limit || g.x == 0 || g.y == 0 || g.z == 0 || g.y > 65535 || g.z > 65535 || b.x * b.y * b.z > 1024) {
        log_op("refused %s dev %d stream %p smem %zu limit %zu", name, g_dev, (void*)st, smem, limit);
        return ret(cudaErrorInvalidValue);
    }
    log_op("launch %s dev %d grid %u %u %u stream %p", name, g_dev, g.x, g.y, g.z, (void*)st);
    return cudaSuccess;
}

}  // namespace

#define L std::lock_guard<std::recursive_mutex> lock(m)

extern "C" {

// ---- the test's side ----
void fake_set(const char* what, int v) {
    L;
    if (!strcmp(what, "clusters")) g_clusters = v;
    if (!strcmp(what, "pinned_failures")) g_pinned_failures = v;
    if (!strcmp(what, "refuse_clusters")) g_refuse_clusters = v;
    if (!strcmp(what, "malloc_failure_at")) g_malloc_failure_at = v;
    if (!strcmp(what, "clear")) g_log.clear();
}
int fake_log_size() { L; return (int)g_log.size(); }
const char* fake_log(int i) { L; return g_log[(size_t)i].c_str(); }

// ---- compiler-generated registration ----
void** __cudaRegisterFatBinary(void*) { static void* h[1]; return h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    L;
    g_names[host] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) { L; g_vars[host] = size; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    L;
    g_calls.push_back({g, b, smem, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    L;
    const Call c = g_calls.back();
    g_calls.pop_back();
    *g = c.grid, *b = c.block, *smem = c.smem, *(cudaStream_t*)st = c.st;
    return cudaSuccess;
}

// ---- devices ----
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { L; *d = g_dev; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { L; g_dev = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof(*p));
    snprintf(p->name, sizeof(p->name), "stand-in");
    p->multiProcessorCount = 148, p->major = 10;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = handle<cudaMemPool_t>(); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { L; const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaDeviceSynchronize(void) { L; log_op("devicesync dev %d", g_dev); return cudaSuccess; }

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) {
    L;
    log_op("malloc bytes %zu", n);
    if (g_malloc_failure_at > 0 && --g_malloc_failure_at == 0) return ret(cudaErrorMemoryAllocation);
    return (*p = malloc(n)) ? cudaSuccess : ret(cudaErrorMemoryAllocation);
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    L;
    if (g_pinned_failures > 0) {
        --g_pinned_failures;
        return ret(cudaErrorMemoryAllocation);
    }
    return cudaMalloc(p, n);
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)180 << 30; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
    L;
    void*& a = g_symbols[{g_dev, s}];
    if (!a) a = calloc(1, g_vars[s]);
    *p = a;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    L;
    log_op("copy %s stream %p bytes %zu",
           k == cudaMemcpyHostToDevice ? "h2d" : k == cudaMemcpyDeviceToHost ? "d2h" : "d2d", (void*)st, n);
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    L;
    log_op("memset stream %p", (void*)st);
    memset(d, v, n);
    return cudaSuccess;
}

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    L;
    *s = handle<cudaStream_t>();
    g_stream_ids[*s] = g_next++;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) {
    L;
    if (g_capturing[s]) {  // as the runtime does: the query ends the capture
        log_op("capture of stream %p invalidated", (void*)s);
        return ret(cudaErrorStreamCaptureUnsupported);
    }
    if (!g_stream_ids.count(s)) g_stream_ids[s] = g_next++;
    *id = g_stream_ids[s];
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { L; log_op("sync stream %p", (void*)s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    L;
    log_op("wait stream %p event %p", (void*)s, (void*)e);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
    L;
    *c = g_capturing[s] ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    L;
    g_capturing[s] = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    L;
    g_capturing[s] = false;
    *g = handle<cudaGraph_t>();
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = handle<cudaGraphExec_t>();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
    L;
    log_op("graph %p stream %p", (void*)e, (void*)s);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { L; *e = handle<cudaEvent_t>(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    L;
    log_op("record stream %p event %p", (void*)s, (void*)e);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

// ---- kernels ----
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    L;
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (v > 227 * 1024) return ret(cudaErrorInvalidValue);
        g_limit[{g_dev, f}] = (size_t)v;
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
    L;
    *n = g_clusters;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t smem, cudaStream_t st) {
    L;
    return launch(f, g, b, smem, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    L;
    for (unsigned i = 0; g_refuse_clusters && i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) return ret(cudaErrorLaunchOutOfResources);
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}
}
