// A CUDA runtime without a device, for tests of the library's host side: device memory is host memory, kernels do
// nothing (their names are logged), and chosen calls fail with the code that the real one would return.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include "internal.h"

namespace {
std::mutex mu;
std::map<char*, size_t> blocks;  // device memory
std::map<const void*, std::string>& names() {  // kernels register from static initialisers
    static std::map<const void*, std::string> m;
    return m;
}
std::string launched;
size_t in_use = 0, budget = (size_t)1 << 40;
int fail_malloc = -1, fail_launch = -1, flag_launch = -1, flags = 0;
thread_local cudaError_t last = cudaSuccess;
thread_local struct { dim3 grid, block; size_t smem; cudaStream_t stream; } config;

cudaError_t set(cudaError_t e) { return e == cudaSuccess ? e : (last = e); }
bool due(int& n) { return n >= 0 && n-- == 0; }

// A traversal that ends with `flags`: written where the launch's parameters point to a control block.
void end_with_flags(void** args) {
    for (int i = 0; i < 64; ++i) {
        char* p = static_cast<char**>(args[0])[i];
        const auto it = blocks.find(p);
        if (it != blocks.end() && it->second == sizeof(c2g::TraversalCtl)) reinterpret_cast<c2g::TraversalCtl*>(p)->flags |= flags;
    }
}

cudaError_t launch(const void* f, void** args, bool coop) {
    std::lock_guard<std::mutex> lk(mu);
    if (coop && due(fail_launch)) return set(cudaErrorLaunchOutOfResources);
    launched += names()[f] + "\n";
    if (coop && due(flag_launch)) end_with_flags(args);
    return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- what the tests set and read
void fake_reset() {
    launched.clear();
    budget = (size_t)1 << 40;
    fail_malloc = fail_launch = flag_launch = -1;
}
void fake_budget(size_t bytes) { budget = bytes; }          // device memory
void fake_fail_malloc(int n) { fail_malloc = n; }           // the n-th cudaMalloc from now is out of memory
void fake_fail_launch(int n) { fail_launch = n; }           // the n-th cooperative launch from now is refused
void fake_flag_launch(int n, int f) { flag_launch = n; flags = f; }  // ... ends with status flags f
size_t fake_in_use() { return in_use; }
const char* fake_launched() { return launched.c_str(); }

// ---- the runtime
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> lk(mu);
    *p = nullptr;
    if (due(fail_malloc) || in_use + n > budget) return set(cudaErrorMemoryAllocation);
    char* m = static_cast<char*>(aligned_alloc(256, (n + 255) / 256 * 256 + 256));
    std::memset(m, 0, n);
    blocks[m] = n;
    in_use += n;
    *p = m;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lk(mu);
    const auto it = blocks.find(static_cast<char*>(p));
    if (!p) return cudaSuccess;
    if (it == blocks.end()) std::abort();  // freed twice
    in_use -= it->second;
    blocks.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = malloc(n), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = malloc(n), cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* p, unsigned) { return *d = p, cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = budget - in_use, *t = budget, cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return n ? memcpy(d, s, n) : d, cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> lk(mu);
    std::memset(a, 0, sizeof(*a));
    auto it = blocks.upper_bound(static_cast<char*>(const_cast<void*>(p)));
    const bool dev = it != blocks.begin() && (--it, static_cast<const char*>(p) < it->first + it->second);
    a->type = dev ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t) { return "fake CUDA error"; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    return *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1, cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { return memset(a, 0, sizeof(*a)), cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 2, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    return *n = 2, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { return *p = const_cast<void*>(s), cudaSuccess; }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) {
    return launch(f, args, true);
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    return *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f)), cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t, cudaStream_t) { return launch(k, args, false); }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
    config.grid = g, config.block = b, config.smem = smem, config.stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = config.grid, *b = config.block, *smem = config.smem, *static_cast<cudaStream_t*>(s) = config.stream;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names()[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

}  // extern "C"
