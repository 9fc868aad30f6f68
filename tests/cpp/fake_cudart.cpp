// A stand-in for the CUDA runtime under the library's host code: device memory
// is host memory, kernels do not run, and every launch is noted with its name
// and shape (the launches of a captured graph when the graph is launched).
// Preloaded ahead of the runtime it shows, without a GPU, which kernels a call
// takes and what the code does when an allocation or an attribute fails.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

namespace {

struct Launch {
    std::string name;
    dim3 grid, block;
    size_t smem;
};
struct Graph {
    std::vector<Launch> launches;
    std::vector<Graph*> bodies;
    cudaGraph_t out[1];
};

std::recursive_mutex mu;
typedef std::lock_guard<std::recursive_mutex> Lock;
std::map<const void*, std::string> names;
std::set<std::pair<int, const void*>> opted_in;  // (device, kernel) with more than 48 KB of dynamic shared memory
std::vector<Launch> log_;
std::map<cudaStream_t, Graph*> capturing;
std::map<void*, size_t> live;
int device = 0, resident = 2, sms = 152;
long allocations = 0, alloc_fails_at = -1, attr_fails_at = -1, launch_fails_at = -1, captures = 0;
thread_local cudaError_t last = cudaSuccess;
thread_local struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} config;

cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
cudaError_t note(const void* f, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    Lock lk(mu);
    if (smem > 48 * 1024 && !opted_in.count({device, f})) return ret(cudaErrorInvalidValue);
    if (launch_fails_at >= 0 && launch_fails_at-- == 0) return ret(cudaErrorLaunchOutOfResources);
    const Launch l{names[f], grid, block, smem};
    auto c = capturing.find(s);
    (c == capturing.end() ? log_ : c->second->launches).push_back(l);
    return cudaSuccess;
}
void replay(const Graph* g) {
    log_.insert(log_.end(), g->launches.begin(), g->launches.end());
    for (const Graph* b : g->bodies) replay(b);
}
int encode_tiled(...) { return 0; }

}  // namespace

extern "C" {

// What the tests set and read.
void fake_set_device(int d) { device = d; }
void fake_set_sms(int n) { sms = n; }
void fake_set_resident(int n) { resident = n; }                     // blocks per SM, shared memory allowing
void fake_fail_allocation(long n) { alloc_fails_at = n < 0 ? -1 : allocations + n; }  // the n-th from now on (0: the next)
void fake_fail_attribute(long n) { attr_fails_at = n; }
void fake_fail_launch(long n) { launch_fails_at = n; }  // (a failed one within a capture ends it)
long fake_allocations(void) { return allocations; }
long fake_live(void) { return (long)live.size(); }
long fake_live_bytes(void) {
    long n = 0;
    for (auto& a : live) n += (long)a.second;
    return n;
}
long fake_captures(void) { return captures; }
void fake_log_clear(void) { log_.clear(); }
int fake_log_size(void) { return (int)log_.size(); }
const char* fake_log_name(int i) { return log_[i].name.c_str(); }
int fake_log_grid(int i) { return (int)(log_[i].grid.x * log_[i].grid.y * log_[i].grid.z); }
int fake_log_block(int i) { return (int)log_[i].block.x; }

void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    Lock lk(mu);
    names[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    config = {grid, block, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(cudaStream_t*)s = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t s) {
    return note((const void*)k, grid, block, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return note(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t s) {
    return note(f, grid, block, smem, s);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int) {
    Lock lk(mu);
    if (attr_fails_at >= 0 && attr_fails_at-- == 0) return ret(cudaErrorInvalidValue);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) opted_in.insert({device, f});
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t smem, unsigned) {
    Lock lk(mu);
    *n = smem > 48 * 1024 && !opted_in.count({device, f}) ? 0 : std::min(resident, (int)(228 * 1024 / (smem + 1024)));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
    *n = 1;
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) {
    Lock lk(mu);
    *p = nullptr;
    if (allocations++ == alloc_fails_at) return ret(cudaErrorMemoryAllocation);
    if (posix_memalign(p, 512, n ? n : 1)) return ret(cudaErrorMemoryAllocation);
    memset(*p, 0, n);
    live[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    Lock lk(mu);
    if (p && !live.erase(p)) return ret(cudaErrorInvalidValue);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemset(void* d, int v, size_t n) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return ret(cudaErrorNotSupported); }

cudaError_t cudaGetDeviceCount(int* n) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = device;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? sms : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError(void) { return last; }
const char* cudaGetErrorName(cudaError_t) { return "fake"; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
    *f = (void*)encode_tiled;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.f;
    return cudaSuccess;
}

cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
    *g = (cudaGraph_t) new Graph();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }  // (an exec is its graph here)
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
    *h = 1;
    return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t g, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                             cudaGraphNodeParams* p) {
    Graph* parent = (Graph*)g;
    Graph* body = new Graph();
    parent->bodies.push_back(body);
    parent->out[0] = (cudaGraph_t)body;
    p->conditional.phGraph_out = parent->out;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
    *x = (cudaGraphExec_t)g;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    Lock lk(mu);
    replay((Graph*)x);
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t s, cudaGraph_t g, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                          size_t, cudaStreamCaptureMode) {
    Lock lk(mu);
    ++captures;
    capturing[s] = (Graph*)g;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode m) {
    return cudaStreamBeginCaptureToGraph(s, (cudaGraph_t) new Graph(), nullptr, nullptr, 0, m);
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    Lock lk(mu);
    *g = (cudaGraph_t)capturing[s];
    capturing.erase(s);
    return cudaSuccess;
}

}  // extern "C"
