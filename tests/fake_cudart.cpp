// A stand-in for the CUDA runtime, preloaded in front of it by
// test_host_runtime.py, so that the host side of libs2dw_cuda.so runs without
// a GPU.  Streams are queues whose operations run when something waits for
// them (so that a copy nobody waited for is still pending), device memory is
// host memory, kernels do nothing but leave a line in a log, and any runtime
// function can be made to fail once at its n-th call.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {

struct Stream {
    int id, prio;
    std::vector<std::pair<bool, std::function<void()>>> ops;  // (is a copy, what it does)
    size_t done = 0;
};
struct Event {
    Stream *s = nullptr;
    size_t pos = 0;
};

Stream g_null{0, 0, {}, 0};
std::vector<Stream *> g_streams{&g_null};
std::map<std::string, int> g_fail;  // calls left before the one that fails
std::map<const void *, std::string> g_names;
std::map<void *, size_t> g_mem, g_pinned;
std::string g_log;
cudaError_t g_last = cudaSuccess;

cudaError_t fails(const char *name, cudaError_t e)
{
    auto it = g_fail.find(name);
    if (it == g_fail.end() || --it->second > 0) return cudaSuccess;
    g_fail.erase(it);
    return g_last = e;
}
#define MAY_FAIL(e)                                              \
    do {                                                         \
        if (fails(__func__, e) != cudaSuccess) return e;         \
    } while (0)

Stream *stream(cudaStream_t s) { return s ? reinterpret_cast<Stream *>(s) : &g_null; }
void drain(Stream *s, size_t to)
{
    while (s->done < to) {
        auto f = s->ops[s->done++].second;
        if (f) f();
    }
}
cudaError_t kernel(const void *f, dim3 g, dim3 b, cudaStream_t st, bool dependent)
{
    Stream *s = stream(st);
    s->ops.push_back({false, {}});
    char line[512];
    snprintf(line, sizeof line, "%d %d %d %s %u,%u,%u %u\n", s->id, s->prio, (int)dependent, g_names[f].c_str(), g.x, g.y,
             g.z, b.x);
    g_log += line;
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- control
void fake_fail(const char *name, int n) { g_fail[name] = n; }
int fake_armed() { return (int)g_fail.size(); }
void fake_pin(void *p, size_t n) { g_pinned[p] = n; }
int fake_pending_copies()
{
    int n = 0;
    for (Stream *s : g_streams)
        for (size_t i = s->done; i < s->ops.size(); i++) n += s->ops[i].first;
    return n;
}
int fake_allocations() { return (int)g_mem.size(); }
// kernel launches since the last call: stream, priority, programmatic, name, grid, block
const char *fake_log()
{
    static std::string out;
    out.swap(g_log);
    g_log.clear();
    return out.c_str();
}

// ---- modules and launches
void **__cudaRegisterFatBinary(void *) { return reinterpret_cast<void **>(&g_null); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    g_names[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
static struct {
    dim3 g, b;
    size_t sm;
    cudaStream_t s;
} g_cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t s)
{
    g_cfg = {g, b, sm, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *sm, void *s)
{
    *g = g_cfg.g;
    *b = g_cfg.b;
    *sm = g_cfg.sm;
    *static_cast<cudaStream_t *>(s) = g_cfg.s;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t, cudaStream_t s)
{
    MAY_FAIL(cudaErrorLaunchOutOfResources);
    return kernel(f, g, b, s, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **)
{
    MAY_FAIL(cudaErrorLaunchOutOfResources);
    bool dep = false;
    for (unsigned i = 0; i < c->numAttrs; i++)
        dep = dep || c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization;
    return kernel(f, c->gridDim, c->blockDim, c->stream, dep);
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 2;
    return cudaSuccess;
}

// ---- device, errors
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *l, int *g) { *l = 0; *g = -5; return cudaSuccess; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }

// ---- memory
cudaError_t cudaMalloc(void **p, size_t n)
{
    MAY_FAIL(cudaErrorMemoryAllocation);
    *p = calloc(n ? n : 1, 1);
    g_mem[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    for (Stream *s : g_streams) drain(s, s->ops.size());
    g_mem.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    MAY_FAIL(cudaErrorMemoryAllocation);
    *p = malloc(n);
    g_pinned[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    g_pinned.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    *a = {};
    a->type = cudaMemoryTypeUnregistered;
    for (auto &q : g_pinned)
        if (p >= q.first && (const char *)p < (char *)q.first + q.second) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    MAY_FAIL(cudaErrorInvalidValue);
    if (!d || !s) return g_last = cudaErrorInvalidValue;
    drain(&g_null, g_null.ops.size());
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    MAY_FAIL(cudaErrorInvalidValue);
    if (!d || !s) return g_last = cudaErrorInvalidValue;
    stream(st)->ops.push_back({true, [=] { memcpy(d, s, n); }});
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n)
{
    if (!p) return g_last = cudaErrorInvalidValue;
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t st)
{
    stream(st)->ops.push_back({false, [=] { memset(p, v, n); }});
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *)
{
    static void *scratch = calloc(40 << 20, 1);
    *p = scratch;
    return cudaSuccess;
}

// ---- streams and events
static cudaError_t new_stream(cudaStream_t *s, int prio)
{
    auto *q = new Stream{(int)g_streams.size(), prio, {}, 0};
    g_streams.push_back(q);
    *s = reinterpret_cast<cudaStream_t>(q);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return new_stream(s, 0); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int prio) { return new_stream(s, prio); }
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    drain(stream(s), stream(s)->ops.size());
    return cudaSuccess;
}
cudaError_t cudaStreamGetPriority(cudaStream_t s, int *p) { *p = stream(s)->prio; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c)
{
    *c = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    MAY_FAIL(cudaErrorUnknown);
    drain(stream(s), stream(s)->ops.size());
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize()
{
    for (Stream *s : g_streams) drain(s, s->ops.size());
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t ev, unsigned)
{
    MAY_FAIL(cudaErrorUnknown);
    const Event e = *reinterpret_cast<Event *>(ev);
    stream(st)->ops.push_back({false, [=] {
                                   if (e.s) drain(e.s, e.pos);
                               }});
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    MAY_FAIL(cudaErrorMemoryAllocation);
    g_log += "event\n";
    *e = reinterpret_cast<cudaEvent_t>(new Event);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    delete reinterpret_cast<Event *>(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    MAY_FAIL(cudaErrorUnknown);
    *reinterpret_cast<Event *>(e) = {stream(s), stream(s)->ops.size()};
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t ev)
{
    Event &e = *reinterpret_cast<Event *>(ev);
    if (e.s) drain(e.s, e.pos);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }

}  // extern "C"
