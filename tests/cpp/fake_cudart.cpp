// A CUDA runtime for tests without a GPU: the library's host code runs
// against it, device memory is host memory and kernels do nothing.  It keeps
// what a device keeps (function attributes, SM counts, capture states) and
// refuses what a device would refuse, and it logs every launch with its
// shape, so that a test can read what the host code decided.
//
// Linked with the library's objects into one shared object (see
// tests/fake_cuda.py); symbols bind inside it.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cxxabi.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

namespace {

struct Launch {
    char name[256];
    int device, grid, block, smem, cooperative, cluster;
    int captured;   // 0 run, 1 recorded into a graph, 2 run by a graph launch
};

struct Stream {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    struct Graph* graph = nullptr;
};
struct Graph {
    std::vector<Launch> launches;
    std::vector<Graph*> bodies;
    bool cooperative() const {
        for (auto& l : launches)
            if (l.cooperative) return true;
        for (auto* b : bodies)
            if (b->cooperative()) return true;
        return false;
    }
};

std::recursive_mutex mu;
int device = 0;
int sms[8] = {148, 100, 148, 148, 148, 148, 148, 148};
int refuse = 0;   // cooperative kernels: 1 refused at launch, 2 in a graph at its instantiation, 4 by the device's attribute
cudaError_t last_error = cudaSuccess;
std::map<const void*, std::string> names;
std::map<std::pair<int, const void*>, int> dyn_smem;
std::set<std::pair<int, const void*>> wide_cluster;
std::map<void*, size_t> device_mem, host_mem;
std::map<const void*, void*> symbols;
std::map<const void*, size_t> symbol_size;
std::vector<Launch> log_;
struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} config;

cudaError_t fail(cudaError_t e) { return last_error = e; }
Stream* at(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
bool real(cudaStream_t s) { return s && s != cudaStreamLegacy && s != cudaStreamPerThread; }

cudaError_t record(const void* f, dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool coop, int cluster) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const auto key = std::make_pair(device, f);
    if (smem > 48 * 1024 && (!dyn_smem.count(key) || dyn_smem[key] < (int)smem)) return fail(cudaErrorInvalidValue);
    if (cluster > 8 && !wide_cluster.count(key)) return fail(cudaErrorInvalidClusterSize);
    const bool capturing = real(s) && at(s)->status == cudaStreamCaptureStatusActive;
    if (coop && ((refuse & 1) && !capturing)) return fail(cudaErrorCooperativeLaunchTooLarge);
    if (coop && (int)grid.x > sms[device]) return fail(cudaErrorCooperativeLaunchTooLarge);
    Launch l{};
    std::snprintf(l.name, sizeof l.name, "%s", names.count(f) ? names[f].c_str() : "?");
    l.device = device;
    l.grid = (int)(grid.x * grid.y * grid.z);
    l.block = (int)block.x;
    l.smem = (int)smem;
    l.cooperative = coop;
    l.cluster = cluster;
    l.captured = capturing;
    if (capturing) at(s)->graph->launches.push_back(l);
    log_.push_back(l);
    return cudaSuccess;
}

CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return CUDA_SUCCESS;
}

}  // namespace

#define API extern "C" __attribute__((visibility("default")))

// ------------------------------------------------------------ for tests --
API void fake_device(int d, int n_sms) {
    device = d;
    if (n_sms > 0) sms[d] = n_sms;
}
API void fake_refuse_cooperative(int how) { refuse = how; }
API void fake_clear_log() { log_.clear(); }
API int fake_launches() { return (int)log_.size(); }
API void fake_launch(int i, Launch* out) { *out = log_[i]; }
API unsigned long long fake_device_bytes() {
    unsigned long long b = 0;
    for (auto& m : device_mem) b += m.second;
    return b;
}
// The live pinned host blocks of a size; returns how many there are.
API int fake_pinned(unsigned long long bytes, void** out, int cap) {
    int n = 0;
    for (auto& m : host_mem)
        if (m.second == bytes) {
            if (n < cap) out[n] = m.first;
            ++n;
        }
    return n;
}

// --------------------------------------------------------- registration --
API void** __cudaRegisterFatBinary(void*) {
    static void* h = nullptr;
    return &h;
}
API void __cudaRegisterFatBinaryEnd(void**) {}
API void __cudaUnregisterFatBinary(void**) {}
API void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    int ok = 0;
    char* d = abi::__cxa_demangle(name, nullptr, nullptr, &ok);
    names[host] = ok == 0 && d ? d : name;
    std::free(d);
}
API void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) { symbol_size[host] = size; }
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, CUstream_st* s) {
    config = {g, b, m, s};
    return 0;
}
API cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = config.grid;
    *b = config.block;
    *m = config.smem;
    *static_cast<cudaStream_t*>(s) = config.stream;
    return cudaSuccess;
}

// --------------------------------------------------------------- device --
API cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
API cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int d) {
    *v = a == cudaDevAttrMultiProcessorCount ? sms[d] : (a == cudaDevAttrCooperativeLaunch ? !(refuse & 4) : 0);
    return cudaSuccess;
}
API cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) { return *a = 0, *b = -1, cudaSuccess; }
API cudaError_t cudaGetLastError() {
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
API const char* cudaGetErrorString(cudaError_t e) {
    return e == cudaErrorInvalidValue ? "invalid argument" : (e == cudaErrorCooperativeLaunchTooLarge ? "too many blocks in cooperative launch" : "error");
}
API cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) dyn_smem[{device, f}] = v;
    if (a == cudaFuncAttributeNonPortableClusterSizeAllowed && v) wide_cluster.insert({device, f});
    return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    const auto key = std::make_pair(device, f);
    if (!wide_cluster.count(key) || !dyn_smem.count(key) || dyn_smem[key] < (int)c->dynamicSmemBytes)
        return fail(cudaErrorInvalidClusterSize);
    *n = 1;
    return cudaSuccess;
}
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t smem, unsigned) {
    const auto key = std::make_pair(device, f);
    *n = smem > 48 * 1024 && (!dyn_smem.count(key) || dyn_smem[key] < (int)smem) ? 0 : 1;
    return cudaSuccess;
}
API cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *p = reinterpret_cast<void*>(&encode);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

// --------------------------------------------------------------- memory --
API cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    std::memset(*p, 0, n);
    device_mem[*p] = n;
    return cudaSuccess;
}
API cudaError_t cudaFree(void* p) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (p && !device_mem.erase(p)) return fail(cudaErrorInvalidValue);
    std::free(p);
    return cudaSuccess;
}
API cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
API cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
API cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    *p = std::calloc(1, n);
    host_mem[*p] = n;
    return cudaSuccess;
}
API cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (p && !host_mem.erase(p)) return fail(cudaErrorInvalidValue);
    std::free(p);
    return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
API cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
API cudaError_t cudaGetSymbolAddress(void** p, const void* sym) {
    if (!symbols.count(sym)) symbols[sym] = std::calloc(1, symbol_size[sym]);
    return *p = symbols[sym], cudaSuccess;
}

// ----------------------------------------------------- streams and events --
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(new Stream()), cudaSuccess;
}
API cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
API cudaError_t cudaStreamDestroy(cudaStream_t s) { return delete at(s), cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = reinterpret_cast<cudaEvent_t>(new int(0)), cudaSuccess; }
API cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
API cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete reinterpret_cast<int*>(e), cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
API cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
API cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }

// ------------------------------------------------------ capture and graphs --
API cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    at(s)->status = cudaStreamCaptureStatusActive;
    at(s)->graph = new Graph();
    return cudaSuccess;
}
API cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t s, cudaGraph_t g, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                                              cudaStreamCaptureMode) {
    at(s)->status = cudaStreamCaptureStatusActive;
    at(s)->graph = reinterpret_cast<Graph*>(g);
    return cudaSuccess;
}
API cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    at(s)->status = cudaStreamCaptureStatusNone;
    *g = reinterpret_cast<cudaGraph_t>(at(s)->graph);
    return cudaSuccess;
}
API cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    return *st = real(s) ? at(s)->status : cudaStreamCaptureStatusNone, cudaSuccess;
}
API cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t s, cudaStreamCaptureStatus* st, unsigned long long* id, cudaGraph_t* g,
                                            const cudaGraphNode_t** deps, size_t* n) {
    *st = at(s)->status;
    if (id) *id = 1;
    if (g) *g = reinterpret_cast<cudaGraph_t>(at(s)->graph);
    if (deps) *deps = nullptr;
    if (n) *n = 0;
    return cudaSuccess;
}
API cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, size_t, unsigned) { return cudaSuccess; }
API cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) { return *h = 1, cudaSuccess; }
API cudaError_t cudaGraphAddNode(cudaGraphNode_t* node, cudaGraph_t g, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
    static std::vector<cudaGraph_t*> outs;
    Graph* body = new Graph();
    reinterpret_cast<Graph*>(g)->bodies.push_back(body);
    outs.push_back(new cudaGraph_t(reinterpret_cast<cudaGraph_t>(body)));
    p->conditional.phGraph_out = outs.back();
    *node = nullptr;
    return cudaSuccess;
}
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    Graph* q = reinterpret_cast<Graph*>(g);
    if ((refuse & 2) && q->cooperative()) return fail(cudaErrorNotSupported);
    *e = reinterpret_cast<cudaGraphExec_t>(new Graph(*q));
    return cudaSuccess;
}
API cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    std::vector<const Graph*> todo{reinterpret_cast<Graph*>(e)};
    while (!todo.empty()) {
        const Graph* g = todo.back();
        todo.pop_back();
        for (Launch l : g->launches) {
            l.captured = 2;
            log_.push_back(l);
        }
        for (auto* b : g->bodies) todo.push_back(b);
    }
    return cudaSuccess;
}
API cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

// -------------------------------------------------------------- launches --
API cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t m, cudaStream_t s) { return record(f, g, b, m, s, false, 1); }
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    bool coop = false;
    int cluster = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i) {
        if (c->attrs[i].id == cudaLaunchAttributeCooperative) coop = c->attrs[i].val.cooperative != 0;
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = (int)c->attrs[i].val.clusterDim.x;
    }
    return record(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream, coop, cluster);
}
