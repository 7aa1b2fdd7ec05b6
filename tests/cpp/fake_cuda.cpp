// fake_cuda.cpp - a host stand-in for the CUDA runtime, linked to the library's objects in tests without a GPU.
// Device memory is host memory, kernels do nothing, and every stream counts the work queued on it.  A buffer of
// a memory pool that is freed while any stream has work that nothing has waited for counts as a violation (the
// runtime's cudaFree does not wait for such a buffer); cudaFree of a plain allocation waits, as the runtime's
// does.  Allocations and queued operations can be made to fail from a given number on.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <vector>

#include "fake_cuda.h"

namespace {

struct Stream {
    uint64_t queued = 0, done = 0;
    std::vector<std::pair<Stream *, uint64_t>> waits;
};
struct Event {
    Stream *stream = nullptr;
    uint64_t at = 0;
};

std::set<Stream *> g_streams;
std::map<void *, std::pair<size_t, bool>> g_live;   // device memory: bytes, of a pool
uint64_t g_pool_allocated = 0;
cudaError_t g_last = cudaSuccess;

void finish(Stream *s, uint64_t at) {
    if (at > s->done) s->done = at;
    for (auto &w : s->waits)
        if (w.second > w.first->done) finish(w.first, w.second);
    s->waits.clear();
}
void finish_all() {
    for (Stream *s : g_streams) finish(s, s->queued);
}
cudaError_t fail(cudaError_t e) {
    ++fake::failed;
    return g_last = e;
}
cudaError_t allocate(void **p, size_t bytes, bool pooled) {
    if (fake::allocations >= fake::fail_allocations_from) return fail(cudaErrorMemoryAllocation);
    ++fake::allocations;
    *p = calloc(1, bytes ? bytes : 1);
    g_live[*p] = {bytes, pooled};
    return cudaSuccess;
}
cudaError_t queue(cudaStream_t stream) {
    if (fake::operations >= fake::fail_operations_from) return fail(cudaErrorUnknown);
    ++fake::operations;
    ++reinterpret_cast<Stream *>(stream)->queued;
    return cudaSuccess;
}

}  // namespace

namespace fake {
uint64_t allocations = 0, operations = 0, launches = 0, violations = 0, failed = 0;
uint64_t fail_allocations_from = ~0ull, fail_operations_from = ~0ull;
uint64_t pool_reserved = 0;
void (*on_copy_out)(void *dst, size_t bytes) = nullptr;
uint64_t pool_used() {
    uint64_t n = 0;
    for (auto &b : g_live) n += b.second.second ? b.second.first : 0;
    return n;
}
size_t live_buffers() { return g_live.size(); }
void reset() {
    finish_all();
    allocations = operations = launches = violations = failed = 0;
    fail_allocations_from = fail_operations_from = ~0ull;
    on_copy_out = nullptr;
    g_last = cudaSuccess;
}
}  // namespace fake

extern "C" {

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { finish_all(); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *free_bytes, size_t *total) { *free_bytes = *total = (size_t)180 << 30; return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t bytes) { return allocate(p, bytes, false); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t, cudaStream_t) {
    const cudaError_t e = allocate(p, bytes, true);
    if (e == cudaSuccess) g_pool_allocated += bytes;
    if (fake::pool_used() > fake::pool_reserved) fake::pool_reserved = fake::pool_used();
    return e;
}
cudaError_t cudaFree(void *p) {
    auto it = g_live.find(p);
    if (it == g_live.end()) return cudaSuccess;
    if (!it->second.second) finish_all();
    for (Stream *s : g_streams) if (s->queued > s->done) { ++fake::violations; break; }
    free(p);
    g_live.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) { *p = calloc(1, bytes ? bytes : 1); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { *p = calloc(1, bytes ? bytes : 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *) {
    *pool = reinterpret_cast<cudaMemPool_t>(0x10);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void *) { return cudaSuccess; }
// (the used bytes that the runtime reports do not go down with cudaFree; cudaFreeAsync is not modelled)
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, enum cudaMemPoolAttr a, void *v) {
    *static_cast<uint64_t *>(v) = a == cudaMemPoolAttrReservedMemCurrent ? fake::pool_reserved : g_pool_allocated;
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t keep) {
    if (fake::pool_reserved > keep) fake::pool_reserved = keep > fake::pool_used() ? keep : fake::pool_used();
    return cudaSuccess;
}

cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind kind, cudaStream_t q) {
    const cudaError_t e = queue(q);
    if (e != cudaSuccess) return e;
    memcpy(d, s, n);
    if (kind == cudaMemcpyDeviceToHost && fake::on_copy_out) fake::on_copy_out(d, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t q) {
    const cudaError_t e = queue(q);
    if (e == cudaSuccess) memset(p, v, n);
    return e;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t q) {
    ++fake::launches;
    return queue(q);
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    Stream *n = new Stream();
    g_streams.insert(n);
    *s = reinterpret_cast<cudaStream_t>(n);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    Stream *n = reinterpret_cast<Stream *>(s);
    finish(n, n->queued);
    for (Stream *o : g_streams) {   // nothing waits for a stream that is gone
        std::vector<std::pair<Stream *, uint64_t>> keep;
        for (auto &w : o->waits) if (w.first != n) keep.push_back(w);
        o->waits.swap(keep);
    }
    g_streams.erase(n);
    delete n;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    Stream *n = reinterpret_cast<Stream *>(s);
    finish(n, n->queued);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    Event *ev = reinterpret_cast<Event *>(e);
    if (ev->stream) reinterpret_cast<Stream *>(s)->waits.push_back({ev->stream, ev->at});
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = reinterpret_cast<cudaEvent_t>(new Event()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    Event *ev = reinterpret_cast<Event *>(e);
    ev->stream = reinterpret_cast<Stream *>(s);
    ev->at = ev->stream->queued;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    Event *ev = reinterpret_cast<Event *>(e);
    if (ev->stream && g_streams.count(ev->stream)) finish(ev->stream, ev->at);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    Event *ev = reinterpret_cast<Event *>(e);
    return !ev->stream || ev->stream->done >= ev->at ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

// graphs are not reached (batches are made with no_graph)
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaErrorUnknown; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorUnknown; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorUnknown; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }

// what the compiler's host code calls around a launch and to register device code
static struct { dim3 grid, block; size_t shared; cudaStream_t stream; } g_call;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sh, cudaStream_t q) { g_call = {g, b, sh, q}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *sh, void *q) {
    *g = g_call.grid;
    *b = g_call.block;
    *sh = g_call.shared;
    *static_cast<cudaStream_t *>(q) = g_call.stream;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
char __cudaInitModule(void **) { return 1; }
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
