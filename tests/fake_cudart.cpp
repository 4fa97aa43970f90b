// A CUDA runtime without a GPU, for host-logic tests: two devices whose memory
// is host memory, kernels that do nothing, and the checks that a launch passes
// on the host side -- above 48 KB of dynamic shared memory a kernel needs its
// limit raised on the device it is launched on.  Wavefront passes end after
// two looks at their counters, the first of which finds 100 paths left.
// libdlgpu.so finds this library in place of libcudart (LD_LIBRARY_PATH).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include "../drawlab_gb300/csrc/internal.h"

namespace {
constexpr int kDevices = 2;
std::recursive_mutex mu;
int device = 0;
cudaError_t last = cudaSuccess;
std::map<const void*, std::string> names;
std::map<const void*, int> limit[kDevices];
std::string log_text, fail_name;
int fail_skip = 0;   // launches of that name that still go through
dl::RenderCounters* counters = nullptr;   // of the pass in progress
unsigned long long total = 0;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} config;

void note(const std::string& s) { log_text += s + "\n"; }

cudaError_t fail(cudaError_t e) { return last = e; }

cudaError_t launch(const void* fn, size_t smem) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const std::string name = names.count(fn) ? names[fn] : "?";
    const int max = limit[device].count(fn) ? limit[device][fn] : 48 * 1024;
    const bool wanted = !fail_name.empty() && name.find(fail_name) != std::string::npos && fail_skip-- <= 0;
    const bool ok = (int)smem <= max && !wanted;
    note((ok ? "launch " : "refused ") + std::to_string(device) + " " + name);
    if (!ok) return fail(wanted ? cudaErrorLaunchOutOfResources : cudaErrorInvalidValue);
    if (name.find("k_init") != std::string::npos && counters) {
        counters->next_path = total;
        counters->ext[0] = 100;
    }
    return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- the test's side
const char* fake_log() { return log_text.c_str(); }
void fake_clear_log() { log_text.clear(); }
void fake_fail_kernel(const char* part_of_name, int skip) {
    fail_name = part_of_name;
    fail_skip = skip;
}

// ---- what compiled CUDA code calls by itself
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names[fn] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
    config = {grid, block, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *static_cast<cudaStream_t*>(st) = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
    *k = (cudaKernel_t)fn;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t smem, cudaStream_t) {
    return launch((const void*)k, smem);
}

// ---- devices, errors, kernels
cudaError_t cudaGetDeviceCount(int* n) { return *n = kDevices, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return device = d, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof(*p));
    p->regsPerMultiprocessor = 65536;
    p->sharedMemPerMultiprocessor = 228 * 1024;
    p->reservedSharedMemPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { return *lo = *hi = 0, cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : "error"; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) limit[device][fn] = v;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->numRegs = 64;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* fn, int, size_t smem, unsigned) {
    *n = (int)smem > (limit[device].count(fn) ? limit[device][fn] : 48 * 1024) ? 0 : 2;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
    return launch(fn, c->dynamicSmemBytes);
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) { return *p = std::calloc(n, 1), *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { return *p = const_cast<void*>(s), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(to, from, n);
    note("copy");
    if (n == 24) {   // a wavefront pass's values, among its counters
        counters = reinterpret_cast<dl::RenderCounters*>(static_cast<char*>(to) - offsetof(dl::RenderCounters, pass_total));
        std::memcpy(&total, from, sizeof(total));
    }
    if (from == counters && n == sizeof(dl::RenderCounters)) counters->ext[0] = 0;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return std::memset(p, v, n), cudaSuccess; }

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)1, cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return *s = (cudaStream_t)2, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return note("wait"), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return note("wait"), cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = (cudaGraph_t)1, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    return *e = (cudaGraphExec_t)1, cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}
