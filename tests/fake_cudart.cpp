// A stand-in for the CUDA runtime, for tests of the library's host side on a
// machine without a GPU: device memory is host memory, a stream is a list of
// copies, fills and frees that run when it is waited for (so that a copy nobody
// waited for can be seen), kernels do nothing, and allocations and cluster
// placement fail where a test asks for it.  Linked with the library's object
// files by test_host_runtime.py.
#include <driver_types.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

namespace {

struct Op {
    char* dst;
    const char* src;  // nullptr: fill with value
    int value;
    size_t n;  // 0: free dst
};
struct Stream {
    std::vector<Op> ops;
};
struct Pool {
    size_t kept = 0, threshold = 0;
};
struct Block {
    size_t n;
    Pool* pool;  // nullptr: none, or the device's default pool
};

std::map<void*, Block> g_blocks;
std::vector<Stream*> g_streams;
size_t g_host_blocks = 0;
std::vector<Pool*> g_pools;
Stream g_default;
size_t g_limit = SIZE_MAX, g_capacity = SIZE_MAX;
int g_max_cluster = 16;
int g_launches_to_error = -1;
bool g_error = false;

Stream* of(cudaStream_t st) { return st ? reinterpret_cast<Stream*>(st) : &g_default; }

void release(void* p) {
    const Block b = g_blocks[p];
    if (b.pool) b.pool->kept += b.n;
    g_blocks.erase(p);
    std::free(p);
}

void drain(Stream* s) {
    for (const Op& o : s->ops) {
        if (!o.n)
            release(o.dst);
        else if (o.src)
            std::memcpy(o.dst, o.src, o.n);
        else
            std::memset(o.dst, o.value, o.n);
    }
    s->ops.clear();
    for (Pool* p : g_pools)
        if (p->kept > p->threshold) p->kept = p->threshold;
}

void drain_all() {
    for (Stream* s : g_streams) drain(s);
    drain(&g_default);
}

int take(void** p, size_t n, Pool* pool) {
    *p = nullptr;
    size_t held = 0;
    for (const auto& b : g_blocks) held += b.second.n;
    for (const Pool* q : g_pools) held += q->kept;
    const size_t reused = pool && pool->kept >= n ? n : 0;
    if (n > g_limit || held - reused + n > g_capacity) return cudaErrorMemoryAllocation;
    *p = std::calloc(1, n ? n : 1);
    g_blocks[*p] = {n, pool};
    if (pool) pool->kept -= pool->kept < n ? pool->kept : n;
    return 0;
}

int context_id(void*, unsigned long long* id) {
    *id = 7;
    return 0;
}

}  // namespace

extern "C" {

// what a test sets and asks
void fake_limit(size_t bytes) { g_limit = bytes; }           // larger device allocations fail
void fake_capacity(size_t bytes) { g_capacity = bytes; }     // of the device, what pools keep included
void fake_refuse_launch(int n) { g_launches_to_error = n; }   // the n-th from here on (0: the next)
void fake_max_cluster(int ctas) { g_max_cluster = ctas; }     // larger clusters cannot be placed
void fake_wait(void) { drain_all(); }                         // for the device
size_t fake_kept(void) {                                      // bytes that pools keep unused
    size_t n = 0;
    for (Pool* p : g_pools) n += p->kept;
    return n;
}
size_t fake_host_blocks(void) { return g_host_blocks; }  // live page-locked allocations
size_t fake_held(void) {  // bytes of live allocations
    size_t n = 0;
    for (const auto& b : g_blocks) n += b.second.n;
    return n;
}
size_t fake_pending(const void* p, size_t n) {  // queued copies from or to [p, p + n)
    const char *a = static_cast<const char*>(p), *b = a + n;
    size_t found = 0;
    for (Stream* s : g_streams)
        for (const Op& o : s->ops)
            found += o.n && ((o.src && o.src < b && o.src + o.n > a) || (o.dst < b && o.dst + o.n > a));
    return found;
}

// memory
int cudaMalloc(void** p, size_t n) { return take(p, n, nullptr); }
int cudaFree(void* p) {
    drain_all();
    if (p) release(p);
    return 0;
}
int cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = std::calloc(1, n);
    ++g_host_blocks;
    return 0;
}
int cudaFreeHost(void* p) {
    drain_all();
    --g_host_blocks;
    std::free(p);
    return 0;
}
int cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n, nullptr); }
int cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
    return take(p, n, reinterpret_cast<Pool*>(pool));
}
int cudaFreeAsync(void* p, cudaStream_t st) {
    of(st)->ops.push_back({static_cast<char*>(p), nullptr, 0, 0});
    return 0;
}
int cudaMemPoolCreate(cudaMemPool_t* out, const cudaMemPoolProps*) {
    g_pools.push_back(new Pool);
    *out = reinterpret_cast<cudaMemPool_t>(g_pools.back());
    return 0;
}
int cudaMemPoolDestroy(cudaMemPool_t pool) {
    for (size_t i = 0; i < g_pools.size(); ++i)
        if (g_pools[i] == reinterpret_cast<Pool*>(pool)) g_pools.erase(g_pools.begin() + (long)i);
    return 0;
}
int cudaMemPoolSetAttribute(cudaMemPool_t pool, int, void* value) {
    reinterpret_cast<Pool*>(pool)->threshold = *static_cast<uint64_t*>(value);
    return 0;
}
int cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep) {
    Pool* p = reinterpret_cast<Pool*>(pool);
    if (p->kept > keep) p->kept = keep;
    return 0;
}
int cudaMemcpyAsync(void* dst, const void* src, size_t n, int, cudaStream_t st) {
    if (n) of(st)->ops.push_back({static_cast<char*>(dst), static_cast<const char*>(src), 0, n});
    return 0;
}
int cudaMemsetAsync(void* dst, int value, size_t n, cudaStream_t st) {
    if (n) of(st)->ops.push_back({static_cast<char*>(dst), nullptr, value, n});
    return 0;
}
int cudaMemcpy(void* dst, const void* src, size_t n, int) {
    drain_all();
    std::memcpy(dst, src, n);
    return 0;
}

// streams and events
int cudaStreamCreateWithFlags(cudaStream_t* out, unsigned) {
    g_streams.push_back(new Stream);
    *out = reinterpret_cast<cudaStream_t>(g_streams.back());
    return 0;
}
int cudaStreamDestroy(cudaStream_t st) {
    drain(of(st));
    for (size_t i = 0; i < g_streams.size(); ++i)
        if (g_streams[i] == of(st)) g_streams.erase(g_streams.begin() + (long)i);
    return 0;
}
int cudaStreamSynchronize(cudaStream_t st) {
    drain(of(st));
    return 0;
}
int cudaStreamQuery(cudaStream_t st) { return cudaStreamSynchronize(st); }
int cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return 0;
}
int cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return 0; }
int cudaEventCreate(cudaEvent_t* e) {
    *e = nullptr;
    return 0;
}
int cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
int cudaEventDestroy(cudaEvent_t) { return 0; }
int cudaEventRecord(cudaEvent_t, cudaStream_t) { return 0; }
int cudaEventSynchronize(cudaEvent_t) { return 0; }

// device, errors, launches
int cudaGetDevice(int* d) {
    *d = 0;
    return 0;
}
int cudaDeviceGetAttribute(int* v, int attr, int) {
    *v = attr == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return 0;
}
int cudaGetDriverEntryPoint(const char* name, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* found) {
    const bool known = std::strcmp(name, "cuCtxGetId") == 0;
    *fn = known ? reinterpret_cast<void*>(context_id) : nullptr;
    *found = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return 0;
}
int cudaGetLastError(void) {
    const int e = g_error ? cudaErrorUnknown : cudaSuccess;
    g_error = false;
    return e;
}
const char* cudaGetErrorString(int) { return "fake error"; }
int cudaFuncSetAttribute(const void*, int, int) { return 0; }
int cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
    int k = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) k = (int)c->attrs[i].val.clusterDim.x;
    *n = k > g_max_cluster ? 0 : 148 / k;
    return 0;
}
int cudaLaunchKernel(void) { return 0; }
int cudaLaunchKernelExC(void) { return 0; }
unsigned __cudaPushCallConfiguration(void) {  // a launch: nothing runs
    if (g_launches_to_error >= 0 && g_launches_to_error-- == 0) g_error = true;
    return 1;
}
int __cudaPopCallConfiguration(void) { return cudaErrorUnknown; }
void** __cudaRegisterFatBinary(void*) {
    static void* handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}

// not reached by these tests
#define CSG_UNUSED(name) \
    int name(void) { return cudaErrorUnknown; }
CSG_UNUSED(cudaEventElapsedTime)
CSG_UNUSED(cudaGetSymbolAddress)
CSG_UNUSED(cudaGraphAddDependencies_v2)
CSG_UNUSED(cudaGraphDestroy)
CSG_UNUSED(cudaGraphExecDestroy)
CSG_UNUSED(cudaGraphGetNodes)
CSG_UNUSED(cudaGraphInstantiate)
CSG_UNUSED(cudaGraphKernelNodeGetParams)
CSG_UNUSED(cudaGraphLaunch)
CSG_UNUSED(cudaGraphNodeGetDependencies)
CSG_UNUSED(cudaGraphNodeGetType)
CSG_UNUSED(cudaStreamBeginCapture)
CSG_UNUSED(cudaStreamEndCapture)
}
