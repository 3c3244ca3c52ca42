// A stand-in for the CUDA runtime, for testing the library's host code without
// a GPU: device memory is host memory, copies and memsets happen at once, and a
// kernel launch checks its configuration and does nothing.  Linked with the
// library's own objects in place of libcudart.
//
// What a test can arrange (fake_* below): how many devices there are, which of
// the coming allocations fail, what counts as pinned memory, and how many
// clusters of a kernel fit.  What it can ask for: launches refused because the
// current device had not been told about their shared memory or cluster size,
// allocations alive, and bytes moved by copies that name plain pageable memory.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <utility>

namespace {

std::mutex mu;
int devices = 1, clusters = 1;
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
long long dev_fail_in = -1;     // device allocations until one fails (once); -1: never
bool pin_fail_always = false, dev_fail_always = false;
std::set<const void *> dev_live;
std::map<const char *, size_t> pin_live;       // pinned ranges
std::map<std::pair<const void *, int>, int> smem_set;
std::set<std::pair<const void *, int>> nonportable;
std::map<const void *, std::string> &names()  // the library's objects register before this file's own are built
{
    static std::map<const void *, std::string> n;
    return n;
}
std::map<std::string, long long> launched;
std::string refused;
long long nrefused = 0, plain_bytes = 0, graph_left = -1;  // graph launches until they fail; -1: never

struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t s;
};
thread_local Config cfg;

cudaError_t err(cudaError_t e)
{
    if (e != cudaSuccess) last = e;
    return e;
}

bool pinned(const void *p)
{
    std::lock_guard<std::mutex> lk(mu);
    auto it = pin_live.upper_bound((const char *)p);
    if (it == pin_live.begin()) return false;
    --it;
    return (const char *)p < it->first + it->second;
}

cudaError_t check_launch(const void *f, dim3 g, dim3 b, size_t smem, unsigned cluster)
{
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(f, current);
    const char *why = nullptr;
    if (smem > 48 * 1024 && (!smem_set.count(key) || (size_t)smem_set[key] < smem)) why = "shared memory";
    else if (cluster > 8 && !nonportable.count(key)) why = "cluster size";
    else if (cluster > 1 && clusters < 1) why = "no cluster fits";
    else if (!g.x || !g.y || !g.z || !b.x || b.x * b.y * b.z > 1024) why = "dimensions";
    if (why) {
        ++nrefused;
        refused = names()[f] + ": " + why;
        return cudaErrorInvalidConfiguration;
    }
    ++launched[names()[f]];
    return cudaSuccess;
}

CUresult fake_encode(CUtensorMap *m, ...)
{
    std::memset(m, 1, sizeof *m);
    return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// ---- what a test arranges and asks ----
void fake_reset(void)
{
    devices = clusters = 1;
    dev_fail_in = -1;
    pin_fail_always = dev_fail_always = false;
    nrefused = plain_bytes = 0;
    graph_left = -1;
    refused.clear();
    launched.clear();
}
void fake_devices(int n) { devices = n; }
void fake_clusters(int n) { clusters = n; }
void fake_fail_device_alloc(long long in) { dev_fail_in = in; }   // 0: the next one
void fake_fail_graph_launch(long long in) { graph_left = in; }
void fake_fail_device(int always) { dev_fail_always = always != 0; }
void fake_fail_pinned(int always) { pin_fail_always = always != 0; }
long long fake_device_live(void) { return (long long)dev_live.size(); }
long long fake_pinned_live(void) { return (long long)pin_live.size(); }
long long fake_plain_bytes(void) { return plain_bytes; }
long long fake_refused(char *buf, size_t n)
{
    if (buf && n) {
        std::strncpy(buf, refused.c_str(), n - 1);
        buf[n - 1] = 0;
    }
    return nrefused;
}
// launches of kernels whose mangled name contains `part`
long long fake_launched(const char *part)
{
    long long n = 0;
    for (auto &k : launched)
        if (k.first.find(part) != std::string::npos) n += k.second;
    return n;
}
void *fake_host_alloc(size_t n)
{
    void *p = nullptr;
    return cudaHostAlloc(&p, n, 0) == cudaSuccess ? p : nullptr;
}
void fake_host_free(void *p) { cudaFreeHost(p); }

// ---- the runtime ----
cudaError_t cudaGetDeviceCount(int *n) { return *n = devices, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d < devices ? (current = d, cudaSuccess) : err(cudaErrorInvalidDevice); }
cudaError_t cudaGetDevice(int *d) { return *d = current, cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int)
{
    std::memset(p, 0, sizeof *p);
    std::strcpy(p->name, "fake");
    p->major = 10;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) { return *p = nullptr, cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}

cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = nullptr;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (dev_fail_in == 0 || dev_fail_always) {
            dev_fail_in = -1;
            return err(cudaErrorMemoryAllocation);
        }
        if (dev_fail_in > 0) --dev_fail_in;
    }
    void *q = std::aligned_alloc(256, (n + 255) / 256 * 256 + 256);
    if (!q) return err(cudaErrorMemoryAllocation);
    std::lock_guard<std::mutex> lk(mu);
    dev_live.insert(q);
    return *p = q, cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    std::lock_guard<std::mutex> lk(mu);
    if (p && !dev_live.erase(p)) std::abort();  // freed twice
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    *p = nullptr;
    if (pin_fail_always) return err(cudaErrorMemoryAllocation);
    char *q = (char *)std::calloc(1, n ? n : 1);
    std::lock_guard<std::mutex> lk(mu);
    pin_live[q] = n ? n : 1;
    return *p = q, cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    std::lock_guard<std::mutex> lk(mu);
    if (p && !pin_live.erase((char *)p)) std::abort();
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    std::memset(a, 0, sizeof *a);
    a->type = pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
    if ((k == cudaMemcpyHostToDevice && !pinned(s)) || (k == cudaMemcpyDeviceToHost && !pinned(d))) {
        std::lock_guard<std::mutex> lk(mu);
        plain_bytes += (long long)n;
    }
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t)
{
    for (size_t i = 0; i < h; ++i) std::memmove((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { return *p = const_cast<void *>(s), cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = (cudaStream_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *,
                                          size_t, cudaStreamCaptureMode)
{
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus *st, unsigned long long *, cudaGraph_t *,
                                        const cudaGraphNode_t **, size_t *)
{
    return *st = cudaStreamCaptureStatusActive, cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned)
{
    return *h = 0, cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t *n, cudaGraph_t, const cudaGraphNode_t *, size_t, cudaGraphNodeParams *p)
{
    static cudaGraph_t body[1] = {};
    p->conditional.phGraph_out = body;
    return *n = nullptr, cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long)
{
    return *e = (cudaGraphExec_t)std::malloc(1), cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t)
{
    if (graph_left == 0) return err(cudaErrorUnknown);
    if (graph_left > 0) --graph_left;
    return cudaSuccess;
}

cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)
{
    std::lock_guard<std::mutex> lk(mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_set[{f, current}] = v;
    if (a == cudaFuncAttributeNonPortableClusterSizeAllowed && v) nonportable.insert({f, current});
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int, size_t smem, unsigned)
{
    std::lock_guard<std::mutex> lk(mu);
    const auto it = smem_set.find({f, current});
    *n = smem > 48 * 1024 && (it == smem_set.end() || (size_t)it->second < smem) ? 0 : 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *)
{
    return *n = clusters, cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t smem, cudaStream_t)
{
    return err(check_launch(f, g, b, smem, 1));
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **)
{
    unsigned cluster = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
    return err(check_launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, cluster));
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **p, unsigned long long, cudaDriverEntryPointQueryResult *q)
{
    *p = std::strcmp(name, "cuTensorMapEncodeTiled") == 0 ? (void *)fake_encode : nullptr;
    *q = *p ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}

unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *s)
{
    cfg = {g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s)
{
    *g = cfg.grid;
    *b = cfg.block;
    *smem = cfg.smem;
    *(cudaStream_t *)s = cfg.s;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *)
{
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, void *, void *, void *, void *, int *)
{
    names()[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
