// A stand-in for the CUDA runtime with which the library's objects are linked
// for CPU tests of its host side: device memory is host memory, kernels do
// nothing, and every launch, copy and fill is written to a log.  Copies to
// the host are held back until something waits for them, so that a test sees
// which are still pending.  Only what the library calls is here.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {
struct Op {
    char kind;            // k kernel, h copy to the host, c other copy, f fill, g graph
    void *stream;
    std::string name;     // of a kernel
    int early;            // programmatic launch attribute
    bool captured;
    unsigned grid, block;
    const void *dst;      // of a copy
    size_t bytes;
};
struct Pending {
    void *stream, *dst;
    const void *src;
    size_t bytes;
};
std::recursive_mutex mu;
std::map<const void *, std::string> names;
std::map<char *, size_t> device, pinned;
std::vector<Op> ops;
std::vector<Pending> pending;
void *capturing = nullptr;
long long copies_left = -1, mallocs_left = -1;   // calls until one fails; -1: none fails
cudaError_t last = cudaSuccess;
int events = 0;
thread_local int current = 0;                    // device
std::map<void *, int> device_of;                 // of streams and events
std::map<void *, void *> recorded;               // event: the stream it was recorded on
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
cudaStream_t cfg_stream;

cudaError_t fail(cudaError_t e) { return last = e; }
void land(void *stream, bool all) {
    for (const Pending &p : pending)
        if (all || p.stream == stream) std::memcpy(p.dst, p.src, p.bytes);
    pending.erase(std::remove_if(pending.begin(), pending.end(), [&](const Pending &p) { return all || p.stream == stream; }),
                  pending.end());
}
bool inside(const std::map<char *, size_t> &m, const void *p) {
    auto it = m.upper_bound((char *)p);
    if (it == m.begin()) return false;
    --it;
    return (const char *)p < it->first + it->second;
}
void log(char kind, void *stream, const std::string &name = "", int early = 0, unsigned grid = 0, unsigned block = 0,
         const void *dst = nullptr, size_t bytes = 0) {
    ops.push_back({kind, stream, name, early, capturing != nullptr && capturing == stream, grid, block, dst, bytes});
}
bool one_fails(long long &left) {
    if (left < 0) return false;
    return left-- == 0;
}
}  // namespace

extern "C" {
// ---- for the test ----
void fake_clear() { std::lock_guard<std::recursive_mutex> l(mu); ops.clear(); }
int fake_ops() { std::lock_guard<std::recursive_mutex> l(mu); return (int)ops.size(); }
int fake_op(int i, char *kind, void **stream, const char **name, int *early, int *captured, unsigned *grid, unsigned *block,
            const void **dst, size_t *bytes) {
    std::lock_guard<std::recursive_mutex> l(mu);
    const Op &o = ops[i];
    *kind = o.kind; *stream = o.stream; *name = o.name.c_str(); *early = o.early; *captured = o.captured;
    *grid = o.grid; *block = o.block; *dst = o.dst; *bytes = o.bytes;
    return 0;
}
int fake_pending() { std::lock_guard<std::recursive_mutex> l(mu); return (int)pending.size(); }
void fake_fail_copy(long long n) { copies_left = n; }
void fake_fail_malloc(long long n) { mallocs_left = n; }
long long fake_pinned_bytes() {
    std::lock_guard<std::recursive_mutex> l(mu);
    long long s = 0;
    for (auto &p : pinned) s += (long long)p.second;
    return s;
}
int fake_live_events() { return events; }

// ---- registration and launches ----
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
    names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
    cfg_grid = g; cfg_block = b; cfg_smem = smem; cfg_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
    *g = cfg_grid; *b = cfg_block; *smem = cfg_smem; *(cudaStream_t *)s = cfg_stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> l(mu);
    log('k', s, names[f], 0, g.x * g.y * g.z, b.x);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
    std::lock_guard<std::recursive_mutex> l(mu);
    int early = 0;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization)
            early = c->attrs[i].val.programmaticStreamSerializationAllowed;
    log('k', c->stream, names[f], early, c->gridDim.x * c->gridDim.y * c->gridDim.z, c->blockDim.x);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    *a = cudaFuncAttributes();
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }

// ---- memory ----
cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (one_fails(mallocs_left)) return fail(cudaErrorMemoryAllocation);
    *p = std::calloc(n ? n : 1, 1);
    device[(char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::recursive_mutex> l(mu);
    land(nullptr, true);
    device.erase((char *)p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    std::lock_guard<std::recursive_mutex> l(mu);
    *p = std::calloc(n ? n : 1, 1);
    pinned[(char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void *p) {
    std::lock_guard<std::recursive_mutex> l(mu);
    land(nullptr, true);
    pinned.erase((char *)p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void *p, size_t n, unsigned) {
    std::lock_guard<std::recursive_mutex> l(mu);
    pinned[(char *)p] = n;
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void *p) {
    std::lock_guard<std::recursive_mutex> l(mu);
    pinned.erase((char *)p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::lock_guard<std::recursive_mutex> l(mu);
    *a = cudaPointerAttributes();
    a->type = inside(device, p) ? cudaMemoryTypeDevice : inside(pinned, p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind k, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (one_fails(copies_left)) return fail(cudaErrorUnknown);
    log(k == cudaMemcpyDeviceToHost ? 'h' : 'c', s, "", 0, 0, 0, dst, n);
    if (k == cudaMemcpyDeviceToHost) {
        pending.push_back({s, dst, src, n});
    } else {
        land(s, false);
        std::memcpy(dst, src, n);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, cudaMemcpyKind k) {
    const cudaError_t e = cudaMemcpyAsync(dst, src, n, k, nullptr);
    std::lock_guard<std::recursive_mutex> l(mu);
    land(nullptr, false);
    return e;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> l(mu);
    land(s, false);
    log('f', s, "", 0, 0, 0, p, n);
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    static double buf[1 << 16];
    *p = buf;
    return cudaSuccess;
}

// ---- devices, streams, events, graphs ----
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 10;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { std::lock_guard<std::recursive_mutex> l(mu); land(nullptr, true); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    std::lock_guard<std::recursive_mutex> l(mu);
    *s = (cudaStream_t)std::malloc(8);
    device_of[*s] = current;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { std::lock_guard<std::recursive_mutex> l(mu); land(s, false); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    std::lock_guard<std::recursive_mutex> l(mu);
    ++events;
    *e = (cudaEvent_t)std::malloc(8);
    device_of[*e] = current;
    recorded.erase(*e);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> l(mu);
    --events;
    std::free(e);
    return cudaSuccess;
}
// an event is recorded on streams of its own device
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (device_of[e] != (s ? device_of[s] : current)) return fail(cudaErrorInvalidResourceHandle);
    recorded[e] = s;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (recorded.count(e)) land(recorded[e], false);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { capturing = s; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { capturing = nullptr; *g = (cudaGraph_t)std::malloc(8); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)std::malloc(8); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { std::free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { std::lock_guard<std::recursive_mutex> l(mu); log('g', s); return cudaSuccess; }
}
