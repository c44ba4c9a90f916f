// A CUDA runtime without a GPU: the calls that the library's host code makes,
// over host memory. Linked with the library's objects it lets tests run the
// host code on the CPU and look at what it asks of the runtime: kernels do
// nothing but are counted and held to the rules that the real runtime has for
// their shared memory and clusters, for each device by itself.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstring>
#include <map>
#include <set>
#include <string>
#include <sys/mman.h>
#include <vector>

namespace {

struct Graph {
    int kernels = 0;           // kernel nodes
    std::vector<Graph*> kids;  // child graphs
    std::vector<Graph*> bodies;
};
struct Stream {
    Graph* capture = nullptr;
};
struct Attributes {
    int dynamic_shared = 48 * 1024;
    bool large_clusters = false;
};
struct Call {
    dim3 grid, block;
    size_t shared;
    cudaStream_t stream;
};

thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
thread_local std::vector<Call> calls;
std::map<std::pair<int, const void*>, Attributes> attributes;
std::map<const void*, std::string> names;
std::map<void*, size_t> blocks;
std::map<std::string, int> executed;  // kernels that ran outside a graph, by name
int executed_total = 0, refused = 0, occupancy_queries = 0;
bool take_clusters = true;
// work that nothing has waited for, on the default stream and on non-blocking
// ones (all that the library makes), and what was done beside it: launches on a
// non-blocking stream, copies and launches on the default one
bool default_stream_busy = false;
std::set<cudaStream_t> busy;
int unordered = 0;
size_t patch_size = 0, patch_offset = 0;
unsigned patch_value = 0;
Stream null_stream;

Stream* of(cudaStream_t s) { return s ? reinterpret_cast<Stream*>(s) : &null_stream; }
cudaError_t keep(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
int all_kernels(const Graph* g) {
    int n = g->kernels;
    for (const auto* k : g->kids) n += all_kernels(k);
    return n;
}

cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t shared, cudaStream_t s, unsigned cluster) {
    const auto it = attributes.find({current, f});
    const Attributes a = it == attributes.end() ? Attributes{} : it->second;
    const bool bad = grid.x == 0 || grid.y == 0 || grid.z == 0 || block.x * block.y * block.z == 0 || block.x * block.y * block.z > 1024;
    if (bad || shared > static_cast<size_t>(a.dynamic_shared) || (cluster > 8 && !a.large_clusters) || (cluster > 1 && grid.x % cluster != 0) || (cluster > 1 && !take_clusters)) {
        ++refused;
        return keep(cudaErrorInvalidValue);
    }
    if (s != nullptr && default_stream_busy) ++unordered;
    if (s == nullptr) {
        if (!busy.empty()) ++unordered;
        default_stream_busy = true;
    }
    if (Graph* g = of(s)->capture) {
        ++g->kernels;
    } else {
        ++executed_total;
        ++executed[names[f]];
        if (s != nullptr) busy.insert(s);
    }
    return cudaSuccess;
}

void copy(void* dst, const void* src, size_t n) {
    std::memcpy(dst, src, n);
    if (n == patch_size) std::memcpy(static_cast<char*>(dst) + patch_offset, &patch_value, sizeof(patch_value));
}

CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }

}  // namespace

extern "C" {

// ---- for the tests ----
void fake_set_device(int d) { current = d; }
int fake_refused() { return refused; }
int fake_occupancy_queries() { return occupancy_queries; }
int fake_unordered() { return unordered; }
int fake_executed() { return executed_total; }
int fake_executed_of(const char* part) {
    int n = 0;
    for (const auto& [name, k] : executed)
        if (name.find(part) != std::string::npos) n += k;
    return n;
}
// launches of clusters fail from now on (false), whatever the queries say
void fake_take_clusters(int yes) { take_clusters = yes != 0; }
// every later copy of exactly `size` bytes arrives with `value` at `offset`:
// what the device would have written there
void fake_patch_copies(size_t size, size_t offset, unsigned value) {
    patch_size = size;
    patch_offset = offset;
    patch_value = value;
}

// ---- registration ----
void** __cudaRegisterFatBinary(void*) {
    static void* handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { names[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t s) {
    calls.push_back({grid, block, shared, s});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* s) {
    const Call c = calls.back();
    calls.pop_back();
    *grid = c.grid;
    *block = c.block;
    *shared = c.shared;
    *static_cast<cudaStream_t*>(s) = c.stream;
    return cudaSuccess;
}

// ---- device, functions, launches ----
cudaError_t cudaGetDevice(int* d) {
    *d = current;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrL2CacheSize ? 126 << 20 : 0);
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    std::strcpy(p->name, "fake");
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    default_stream_busy = false;
    busy.clear();
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    Attributes& t = attributes[{current, f}];
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) t.dynamic_shared = v;
    else if (a == cudaFuncAttributeNonPortableClusterSizeAllowed) t.large_clusters = v != 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    ++occupancy_queries;
    const Attributes a = attributes[{current, f}];
    const unsigned size = c->numAttrs > 0 ? c->attrs[0].val.clusterDim.x : 1;
    *n = c->dynamicSmemBytes <= static_cast<size_t>(a.dynamic_shared) && (size <= 8 || a.large_clusters) ? 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t shared, cudaStream_t s) { return launch(f, grid, block, shared, s, 1); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    unsigned cluster = 1;
    for (unsigned k = 0; k < c->numAttrs; ++k)
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[k].val.clusterDim.x;
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream, cluster);
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
    *p = const_cast<void*>(symbol);
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *p = reinterpret_cast<void*>(&encode);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) {
    void* m = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return keep(cudaErrorMemoryAllocation);
    blocks[m] = n ? n : 1;
    *p = m;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p == nullptr) return cudaSuccess;
    const auto it = blocks.find(p);
    if (it == blocks.end()) return keep(cudaErrorInvalidValue);
    munmap(p, it->second);
    blocks.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (of(st)->capture == nullptr) copy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (!busy.empty()) ++unordered;
    copy(d, s, n);
    return cudaSuccess;
}
// fresh memory is zero already: clearing the large blocks would only touch them
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s) {
    if (s == nullptr) default_stream_busy = true;
    if (of(s)->capture == nullptr && n <= (1u << 20)) std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }  // returns before it has run

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(new Stream);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    delete of(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (s == nullptr) default_stream_busy = false;
    busy.erase(s);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    of(s)->capture = new Graph;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t s, cudaGraph_t g, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, cudaStreamCaptureMode) {
    of(s)->capture = reinterpret_cast<Graph*>(g);
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    *g = reinterpret_cast<cudaGraph_t>(of(s)->capture);
    of(s)->capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = of(s)->capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, cudaStreamCaptureStatus* st, unsigned long long*, cudaGraph_t* g, const cudaGraphNode_t** deps, size_t* n) {
    cudaStreamIsCapturing(s, st);
    if (g) *g = reinterpret_cast<cudaGraph_t>(of(s)->capture);
    if (deps) *deps = nullptr;
    if (n) *n = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(new int(0));
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete reinterpret_cast<int*>(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
    *g = reinterpret_cast<cudaGraph_t>(new Graph);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphAddChildGraphNode(cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t*, size_t, cudaGraph_t child) {
    *n = nullptr;
    reinterpret_cast<Graph*>(g)->kids.push_back(reinterpret_cast<Graph*>(child));
    return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
    *n = nullptr;
    Graph* const body = new Graph;
    reinterpret_cast<Graph*>(g)->bodies.push_back(body);
    static cudaGraph_t out[1];
    out[0] = reinterpret_cast<cudaGraph_t>(body);
    p->conditional.phGraph_out = out;
    return cudaSuccess;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
    *h = 1;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    executed_total += all_kernels(reinterpret_cast<Graph*>(e));
    return cudaSuccess;
}

}  // extern "C"
