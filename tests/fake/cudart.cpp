// A stand-in for the CUDA runtime that the host code's tests link the library's
// objects against (test_host_faults.py): two devices without any kernel
// execution.  Device memory is host memory, copies are memcpy, kernels are
// recorded by name and do nothing, graphs and captures are refused.
//
// Refusals and delays, set by the tests:
//   fake_refuse(text)    launches of kernels whose name contains text fail
//   fake_busy(ms)        an event is done that long after its record
//   fake_context(id)     the current context; memory of another one is refused
//   fake_launches(text, device)  accepted launches so far (device < 0: all)
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <chrono>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

namespace {

using Clock = std::chrono::steady_clock;

struct Launch {
    std::string name;
    int device;
};
struct Block {
    size_t n;
    bool host;
    unsigned long long context;
};
struct Event {
    Clock::time_point done{};
};
struct Call {
    dim3 grid, block;
    size_t smem;
    void* stream;
};

std::mutex mu;
// host stub -> name; the objects register theirs before this file's globals exist
std::map<const void*, std::string>& kernels() {
    static std::map<const void*, std::string> m;
    return m;
}
std::map<std::pair<int, const void*>, bool> large;     // non-portable clusters allowed
std::map<const char*, Block> blocks;  // by address
unsigned long long context = 1;
std::vector<Launch> launches;
std::string refuse;
int busy_ms = 0;
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
thread_local std::vector<Call> calls;

cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
cudaError_t launch(const void* f, unsigned cluster) {
    std::lock_guard<std::mutex> l(mu);
    const std::string& name = kernels()[f];
    if (!refuse.empty() && name.find(refuse) != std::string::npos)
        return set(cudaErrorLaunchOutOfResources);
    if (cluster > 8 && !large[{current, f}]) return set(cudaErrorInvalidClusterSize);
    launches.push_back({name, current});
    return cudaSuccess;
}
cudaError_t take(void** p, size_t n, bool host) {
    *p = std::calloc(n ? n : 1, 1);
    std::lock_guard<std::mutex> l(mu);
    blocks[(const char*)*p] = {n, host, context};
    return cudaSuccess;
}
cudaError_t give(void* p) {
    if (!p) return cudaSuccess;
    {
        std::lock_guard<std::mutex> l(mu);
        if (!blocks.erase((const char*)p)) return set(cudaErrorInvalidValue);
    }
    std::free(p);
    return cudaSuccess;
}
cudaError_t copy(void* d, const void* s, size_t n) {
    {
        std::lock_guard<std::mutex> l(mu);
        for (const char* p : {(const char*)d, (const char*)s}) {
            auto it = blocks.upper_bound(p);
            if (it == blocks.begin() || p >= (--it)->first + it->second.n) continue;
            if (!it->second.host && it->second.context != context)
                return set(cudaErrorInvalidValue);
        }
    }
    std::memcpy(d, s, n);
    return cudaSuccess;
}
int context_id(void*, unsigned long long* id) {
    *id = context;
    return 0;
}
unsigned cluster_of(const cudaLaunchConfig_t* c) {
    for (unsigned q = 0; q < c->numAttrs; q++)
        if (c->attrs[q].id == cudaLaunchAttributeClusterDimension)
            return c->attrs[q].val.clusterDim.x * c->attrs[q].val.clusterDim.y *
                   c->attrs[q].val.clusterDim.z;
    return 1;
}

}  // namespace

extern "C" {

void fake_refuse(const char* text) {
    std::lock_guard<std::mutex> l(mu);
    refuse = text;
}
void fake_context(unsigned long long id) {
    std::lock_guard<std::mutex> l(mu);
    context = id;
}
void fake_busy(int ms) { busy_ms = ms; }
int fake_launches(const char* text, int device) {
    std::lock_guard<std::mutex> l(mu);
    int n = 0;
    for (const Launch& q : launches)
        n += q.name.find(text) != std::string::npos && (device < 0 || q.device == device);
    return n;
}

// what the compiler's host code calls (crt/host_runtime.h)
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
    kernels()[stub] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
    calls.push_back({g, b, smem, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    const Call c = calls.back();
    calls.pop_back();
    *g = c.grid;
    *b = c.block;
    *smem = c.smem;
    *(void**)st = c.stream;
    return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) {
    return launch(f, 1);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return launch(f, cluster_of(c));
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    std::lock_guard<std::mutex> l(mu);
    if (a == cudaFuncAttributeNonPortableClusterSizeAllowed) large[{current, f}] = v != 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    std::lock_guard<std::mutex> l(mu);
    *n = cluster_of(c) <= 8 || large[{current, f}] ? 4 : 0;
    return *n ? cudaSuccess : set(cudaErrorInvalidClusterSize);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int,
                                                                   size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = current;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d > 1) return set(cudaErrorInvalidDevice);
    current = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t) { return "refused by the stand-in"; }

cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, false); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return take(p, n, true); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeHost(void* p) { return give(p); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    std::lock_guard<std::mutex> l(mu);
    auto it = blocks.upper_bound((const char*)p);
    if (it != blocks.begin() && (const char*)p < (--it)->first + it->second.n)
        a->type = it->second.host ? cudaMemoryTypeHost : cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return copy(d, s, n);
}
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long,
                                    cudaDriverEntryPointQueryResult* r) {
    const bool known = !std::strcmp(name, "cuCtxGetId");
    *f = known ? (void*)context_id : nullptr;
    if (r) *r = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return set(cudaErrorInvalidSymbol); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free((void*)s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }

cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t) new Event;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete (Event*)e;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    ((Event*)e)->done = Clock::now() + std::chrono::milliseconds(busy_ms);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    return Clock::now() < ((Event*)e)->done ? set(cudaErrorNotReady) : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::this_thread::sleep_until(((Event*)e)->done);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.0f;
    return cudaSuccess;
}

// no graphs
cudaError_t cudaGraphCreate(cudaGraph_t*, unsigned) { return set(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) {
    return set(cudaErrorNotSupported);
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return set(cudaErrorNotSupported); }
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t,
                             cudaGraphNodeParams*) {
    return set(cudaErrorNotSupported);
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned,
                                             unsigned) {
    return set(cudaErrorNotSupported);
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    return set(cudaErrorNotSupported);
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*,
                                          const cudaGraphEdgeData*, size_t,
                                          cudaStreamCaptureMode) {
    return set(cudaErrorNotSupported);
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = nullptr;
    return set(cudaErrorNotSupported);
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus* s,
                                     unsigned long long*, cudaGraph_t*, const cudaGraphNode_t**,
                                     size_t*) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, size_t, unsigned) {
    return set(cudaErrorNotSupported);
}

}  // extern "C"
