// The CUDA runtime calls of the engine's host code (csrc/host.cpp) on host
// memory, for tests without a GPU: device memory is the heap, work on a stream
// runs at once, and every call is written to a log.  A chosen call can be made
// to fail, and handles are checked: one that was never made or is gone is an
// error.  Kernels are left out (outputs are whatever the memory holds).
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>

#include "engine.h"

namespace {

std::recursive_mutex lock;
std::set<void *> streams, events;
std::map<char *, size_t> device, pinned;
std::string log_text, fail_name;
int fail_after = -1;
long next_handle = 0x1000;
std::map<void *, int> ids;

void note(const std::string &s) { log_text += s + "\n"; }
bool failing(const char *name) {
    if (fail_after < 0 || fail_name != name) return false;
    return fail_after-- == 0;
}
std::string id(void *h) { return h ? std::to_string(ids[h]) : "0"; }
void *handle(std::set<void *> &of) {
    void *h = reinterpret_cast<void *>(next_handle += 16);
    ids[h] = (int)ids.size() + 1;
    of.insert(h);
    return h;
}
// the legacy default stream is no handle of ours
cudaError_t on(cudaStream_t s) {
    if (!s || streams.count(s)) return cudaSuccess;
    note("bad stream");
    return cudaErrorInvalidResourceHandle;
}
cudaError_t known(cudaEvent_t e) {
    if (events.count(e)) return cudaSuccess;
    note("bad event");
    return cudaErrorInvalidResourceHandle;
}
bool within(const std::map<char *, size_t> &m, const void *p) {
    auto it = m.upper_bound((char *)p);
    if (it == m.begin()) return false;
    --it;
    return (const char *)p < it->first + it->second;
}
std::string side(const void *p) { return within(device, p) ? "device" : within(pinned, p) ? "pinned" : "host"; }

}  // namespace

#define BEGIN(name)                                                \
    std::lock_guard<std::recursive_mutex> guard(lock);             \
    if (failing(name)) return cudaErrorMemoryAllocation

extern "C" {
void fake_reset() { log_text.clear(); fail_after = -1; }
void fake_fail(const char *name, int after) { fail_name = name; fail_after = after; }
const char *fake_log() { return log_text.c_str(); }
long fake_live(int kind) { return (long)(kind == 0 ? streams.size() : kind == 1 ? events.size() : kind == 2 ? device.size() : pinned.size()); }

cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "injected"; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) { std::memset(p, 0, sizeof *p); p->major = 10; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { BEGIN("cudaStreamCreateWithFlags"); *s = (cudaStream_t)handle(streams); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { BEGIN("cudaStreamDestroy"); return streams.erase(s) ? cudaSuccess : (note("bad stream"), cudaErrorInvalidResourceHandle); }
cudaError_t cudaStreamQuery(cudaStream_t s) { BEGIN("cudaStreamQuery"); return on(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { BEGIN("cudaStreamSynchronize"); note("wait stream " + id(s)); return on(s); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { BEGIN("cudaStreamWaitEvent"); return on(s) ? on(s) : known(e); }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }

cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { BEGIN("cudaEventCreateWithFlags"); *e = (cudaEvent_t)handle(events); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { BEGIN("cudaEventDestroy"); return events.erase(e) ? cudaSuccess : (note("bad event"), cudaErrorInvalidResourceHandle); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { BEGIN("cudaEventRecord"); note("record " + id(e) + " on " + id(s)); return known(e) ? known(e) : on(s); }
cudaError_t cudaEventQuery(cudaEvent_t e) { BEGIN("cudaEventQuery"); return known(e); }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { BEGIN("cudaEventSynchronize"); note("wait event " + id(e)); return known(e); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n) { BEGIN("cudaMalloc"); *p = std::calloc(n + 256, 1); device[(char *)*p] = n; return cudaSuccess; }
cudaError_t cudaFree(void *p) { BEGIN("cudaFree"); device.erase((char *)p); std::free(p); return cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) {
    BEGIN("cudaMallocAsync");
    if (on(s)) return on(s);
    *p = std::aligned_alloc(256, (n + 511) / 256 * 256);
    std::memset(*p, 0, n);
    device[(char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { BEGIN("cudaFreeAsync"); if (on(s)) return on(s); device.erase((char *)p); std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { BEGIN("cudaHostAlloc"); *p = std::aligned_alloc(4096, (n + 4095) / 4096 * 4096); pinned[(char *)*p] = n; return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { BEGIN("cudaFreeHost"); pinned.erase((char *)p); std::free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { BEGIN("cudaMemset"); std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) { BEGIN("cudaMemsetAsync"); std::memset(p, v, n); return on(s); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { BEGIN("cudaMemcpy"); note("copy " + side(s) + " to " + side(d) + " " + std::to_string(n)); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    BEGIN("cudaMemcpyAsync");
    note("copy " + side(s) + " to " + side(d) + " " + std::to_string(n) + " on " + id(st));
    std::memcpy(d, s, n);
    return on(st);
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::lock_guard<std::recursive_mutex> guard(lock);
    std::memset(a, 0, sizeof *a);
    a->type = within(device, p) ? cudaMemoryTypeDevice : within(pinned, p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
}  // extern "C"

namespace jxr {
size_t tile_smem_bytes(int) { return 0; }
int tile_mbs() { return 4; }
cudaError_t launch_tiles(const ImageDev *, const void *, const uint32_t *, uint32_t, int, uint32_t *, uint32_t *,
                         const cudaStream_t *lanes, int lane_count, const LaunchTuning *) {
    BEGIN("launch_tiles");
    note("launch on " + std::to_string(lane_count));
    for (int k = 0; k < lane_count; k++)
        if (on(lanes[k])) return on(lanes[k]);
    return cudaSuccess;
}
cudaError_t launch_quarter(const ImageDev *, const QuarterImage *, uint32_t, const QuarterPlane *, uint32_t, bool, bool,
                           bool, uint32_t, uint32_t, uint64_t, uint32_t *, cudaStream_t stream) {
    BEGIN("launch_quarter");
    return on(stream);
}
}  // namespace jxr
