// A stand-in for the CUDA runtime that the library's objects link against, so that
// its host code runs without a GPU and any runtime call can be made to fail: see
// fake_cudart.h.  Only what the library calls is here.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

namespace {

struct State {
    std::map<const char *, size_t> dev;  // device allocations
    std::map<const char *, size_t> pinned;
    std::map<const void *, std::string> kernels;
    std::map<const void *, void *> symbols;
    std::map<const void *, size_t> symbol_bytes;
    std::vector<std::pair<std::string, int>> watched;
    std::vector<fake::Launch> launches;
    std::map<const char *, size_t> flying;  // null-stream transfers not yet waited for
    std::map<std::string, fake::SmemLimit> smem;
    int n_malloc = 0, n_graph = 0, n_early = 0, n_wait = 0, capturing = 0, fail_malloc = 0, fail_upload = 0, fail_inst = 0;
    bool malloc_after = false, inst_after = false;
    cudaError_t last = cudaSuccess;
    size_t handle = 0x1000;
};
State &S() {
    static State *s = new State();  // outlives the objects' own static state
    return *s;
}

cudaError_t err(cudaError_t e) {
    if (e != cudaSuccess) S().last = e;
    return e;
}
bool due(int &n, bool after = false) {
    if (n <= 0) return false;
    if (n == 1) {
        if (!after) n = 0;
        return true;
    }
    --n;
    return false;
}
const std::pair<const char *const, size_t> *find(const std::map<const char *, size_t> &m, const void *p) {
    auto it = m.upper_bound((const char *)p);
    if (it == m.begin()) return nullptr;
    --it;
    return (const char *)p < it->first + it->second ? &*it : nullptr;
}
bool device_range(const void *p, size_t n) {
    auto *a = find(S().dev, p);
    if (a && (const char *)p + n <= a->first + a->second) return true;
    for (auto &s : S().symbols) {
        const char *b = (const char *)s.second;
        if ((const char *)p >= b && (const char *)p + n <= b + S().symbol_bytes[s.first]) return true;
    }
    return false;
}
cudaError_t copy(void *d, const void *s, size_t n, cudaMemcpyKind k, bool null_stream) {
    if (!n) return cudaSuccess;
    if (k == cudaMemcpyHostToDevice && due(S().fail_upload)) return err(cudaErrorInvalidValue);
    const bool d_dev = find(S().dev, d) != nullptr, s_dev = find(S().dev, s) != nullptr;
    const bool to_dev = k == cudaMemcpyHostToDevice || k == cudaMemcpyDeviceToDevice;
    const bool from_dev = k == cudaMemcpyDeviceToHost || k == cudaMemcpyDeviceToDevice;
    if (to_dev != (d_dev || device_range(d, 1)) || from_dev != (s_dev || device_range(s, 1)))
        return err(cudaErrorInvalidValue);
    if ((to_dev && !device_range(d, n)) || (from_dev && !device_range(s, n))) {
        fprintf(stderr, "fake: copy out of range\n");
        abort();
    }
    memmove(d, s, n);
    if (null_stream && k == cudaMemcpyHostToDevice && !find(S().pinned, s)) S().flying[(const char *)d] = n;
    if (k == cudaMemcpyDeviceToHost && null_stream) S().flying.clear();
    return cudaSuccess;
}
template <typename T>
cudaError_t make(T *out) {
    *out = (T)(S().handle += 0x10);
    return cudaSuccess;
}
void record(const void *fn, dim3 grid, void **args, cudaStream_t st) {
    fake::Launch l{S().kernels.count(fn) ? S().kernels[fn] : "?", st, grid.x * grid.y * grid.z, {}, false};
    for (auto &w : S().watched)
        if (l.name.find(w.first) != std::string::npos) {
            l.ptr.push_back(*(const void **)args[w.second]);
            l.early = l.early || (st && find(S().flying, l.ptr.back()));
        }
    if (st && !S().capturing && !S().flying.empty()) ++S().n_early;
    S().launches.push_back(l);
}
struct Config {
    dim3 g, b;
    size_t smem;
    cudaStream_t st;
};
Config g_cfg;
int encode_stub(...) { return 0; }
int ctx_stub(void **p) {
    *p = (void *)0x77;
    return 0;
}
int ctx_id_stub(void *, unsigned long long *id) {
    *id = 7;
    return 0;
}

}  // namespace

namespace fake {
void fail_malloc(int n, bool after) { S().fail_malloc = n, S().malloc_after = after; }
void fail_upload(int n) { S().fail_upload = n; }
void fail_instantiate(int n, bool after) { S().fail_inst = n, S().inst_after = after; }
int stream_waits() { return S().n_wait; }
int graph_launches() { return S().n_graph; }
int early_launches() { return S().n_early; }
int mallocs() { return S().n_malloc; }
size_t live_bytes() {
    size_t t = 0;
    for (auto &a : S().dev) t += a.second;
    return t;
}
bool is_device(const void *p) { return find(S().dev, p) != nullptr; }
void *device_only(size_t bytes) {
    void *p = mmap(nullptr, bytes, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    S().dev[(const char *)p] = bytes;
    return p;
}
void watch(const char *k, int arg) { S().watched.push_back({k, arg}); }
std::vector<Launch> take_launches() {
    std::vector<Launch> l;
    l.swap(S().launches);
    return l;
}
SmemLimit smem_limit(const char *k) {
    for (auto &s : S().smem)
        if (s.first.find(k) != std::string::npos) return s.second;
    return {};
}
}  // namespace fake

extern "C" {

// ---- registration and launches ------------------------------------------------
void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    S().kernels[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) {
    S().symbols[host] = calloc(1, size);
    S().symbol_bytes[host] = size;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *st) {
    g_cfg = {g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
    *g = g_cfg.g;
    *b = g_cfg.b;
    *smem = g_cfg.smem;
    *(cudaStream_t *)st = g_cfg.st;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) {
    *k = (cudaKernel_t)fn;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void **args, size_t, cudaStream_t st) {
    record((const void *)k, grid, args, st);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args) {
    record(fn, c->gridDim, args, c->stream);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
    *p = S().symbols[sym];
    return *p ? cudaSuccess : err(cudaErrorInvalidSymbol);
}
cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        auto &s = S().smem[S().kernels[fn]];
        s.last = v;
        if (v > s.most) s.most = v;
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}

// ---- device and errors ----------------------------------------------------------
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof(*p));
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) {
    *lo = 0;
    *hi = -5;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    S().flying.clear();
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = S().last;
    S().last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q) {
    *p = !strcmp(name, "cuCtxGetCurrent") ? (void *)ctx_stub
         : !strcmp(name, "cuCtxGetId")    ? (void *)ctx_id_stub
                                          : (void *)encode_stub;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

// ---- memory -----------------------------------------------------------------------
cudaError_t cudaMalloc(void **p, size_t n) {
    ++S().n_malloc;
    *p = nullptr;
    if (due(S().fail_malloc, S().malloc_after)) return err(cudaErrorMemoryAllocation);
    *p = calloc(1, n ? n : 1);
    S().dev[(const char *)*p] = n ? n : 1;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (!p) return cudaSuccess;
    if (!S().dev.count((const char *)p)) {
        fprintf(stderr, "fake: free of what was not allocated\n");
        abort();
    }
    S().dev.erase((const char *)p);
    S().flying.erase((const char *)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
    *p = calloc(1, n);
    S().pinned[(const char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    S().pinned.erase((const char *)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    memset(a, 0, sizeof(*a));
    a->type = find(S().dev, p) ? cudaMemoryTypeDevice
              : find(S().pinned, p) ? cudaMemoryTypeHost
                                    : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k, true); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    return copy(d, s, n, k, st == nullptr);
}
static cudaError_t set(void *d, int v, size_t n, bool null_stream) {
    if (!n) return cudaSuccess;
    if (!device_range(d, n)) return err(cudaErrorInvalidValue);
    memset(d, v, n);
    if (null_stream) S().flying[(const char *)d] = n;
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return set(d, v, n, true); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { return set(d, v, n, st == nullptr); }

// ---- streams, events, graphs ------------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return make(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return make(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    ++S().n_wait;
    if (!st) S().flying.clear();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return make(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return make(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    S().flying.clear();
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    ++S().capturing;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *,
                                          size_t, cudaStreamCaptureMode) {
    ++S().capturing;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    --S().capturing;
    return make(g);
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus *s, unsigned long long *, cudaGraph_t *g,
                                     const cudaGraphNode_t **d, const cudaGraphEdgeData **e, size_t *n) {
    *s = cudaStreamCaptureStatusActive;
    if (g) make(g);
    if (d) *d = nullptr;
    if (e) *e = nullptr;
    if (n) *n = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                                                unsigned) {
    return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t *n, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                             cudaGraphNodeParams *p) {
    static cudaGraph_t bodies[8];
    if (p->type == cudaGraphNodeTypeConditional) p->conditional.phGraph_out = bodies;
    return make(n);
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) {
    return make(h);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    *e = nullptr;
    if (due(S().fail_inst, S().inst_after)) return err(cudaErrorMemoryAllocation);
    return make(e);
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t st) {
    ++S().n_graph;
    if (st && !S().flying.empty()) ++S().n_early;
    return e ? cudaSuccess : err(cudaErrorInvalidValue);
}

}  // extern "C"
