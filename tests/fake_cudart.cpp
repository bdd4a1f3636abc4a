// A stand-in for the CUDA runtime, for tests of the library's host code on a
// machine without a GPU: the library's objects are linked against this file.
// Device memory is host memory that starts as zeros, kernels do not run, and
// what the library asks of the runtime is recorded:
//   - a host-to-device copy or fill on the legacy stream counts as under way
//     until that stream is waited for, and a kernel launched on another stream
//     meanwhile is noted as unordered;
//   - cudaMalloc's sizes are noted, and it can be made to fail;
//   - a launch asking for more dynamic shared memory than the kernel's
//     attribute allows is refused.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>

namespace {
std::recursive_mutex mu;
std::map<const void*, std::string> names;  // kernels by their host stub
std::map<const void*, int> smemAttr;       // their dynamic shared memory limits
std::map<void*, size_t> live;              // device allocations
std::string events;
int sms = 148, failIn = 0, mallocs = 0;
bool legacyPending = false;
cudaError_t lastError = cudaSuccess;
thread_local std::vector<std::tuple<dim3, dim3, size_t, void*>> configs;

cudaError_t fail(cudaError_t e) { return lastError = e; }
void note(const std::string& s) { events += s + "\n"; }
int limitOf(const void* fn) { return smemAttr.count(fn) ? smemAttr[fn] : 48 * 1024; }

cudaError_t launched(const void* fn, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    const std::string& n = names[fn];
    std::ostringstream o;
    o << "launch " << n << " grid " << g.x << " block " << b.x << " smem " << smem;
    // packTilesKernel's seventh argument: the columns to write, or null
    if (n.find("packTilesKernel") != std::string::npos) o << " columns " << (*static_cast<void**>(args[6]) ? 1 : 0);
    note(o.str());
    if (s && legacyPending) note("unordered " + n);
    if ((int)smem > limitOf(fn)) {
        note("refused " + n);
        return fail(cudaErrorInvalidValue);
    }
    return cudaSuccess;
}
cudaError_t copy(void* d, const void* s, size_t n) {
    if (n) std::memcpy(d, s, n);
    return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- what the tests call ----
void fake_device(int multiprocessors) { sms = multiprocessors; }
void fake_reset() {
    std::lock_guard<std::recursive_mutex> lock(mu);
    events.clear();
    failIn = mallocs = 0;
    legacyPending = false;
}
const char* fake_events() { return events.c_str(); }
void fake_fail_malloc(int nth) { failIn = nth; }  // the nth cudaMalloc from here fails; 0: none
int fake_mallocs() { return mallocs; }            // since the reset
int fake_live() { return (int)live.size(); }

// ---- registration and launches ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { names[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) { configs.emplace_back(g, b, smem, s); return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    std::tie(*g, *b, *smem, *static_cast<void**>(s)) = configs.back();
    configs.pop_back();
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t smem, cudaStream_t s) { return launched(f, g, b, a, smem, s); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** a, size_t smem, cudaStream_t s) { return launched(f, g, b, a, smem, s); }

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    ++mallocs;
    note("malloc " + std::to_string(n));
    if (failIn && --failIn == 0) return fail(cudaErrorMemoryAllocation);
    *p = std::calloc(std::max<size_t>(n, 1), 1);
    live[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    if (!p) return cudaSuccess;
    if (!live.erase(p)) { note("bad free"); return fail(cudaErrorInvalidValue); }
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
    legacyPending = k == cudaMemcpyHostToDevice;  // a copy to the host waits for what is before it
    return copy(d, s, n);
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (!st) legacyPending = true;
    return copy(d, s, n);
}
cudaError_t cudaMemset(void* d, int v, size_t n) { legacyPending = true; std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    if (!st) legacyPending = true;
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char scratch[16 << 20]; *p = scratch; return cudaSuccess; }

// ---- streams, events, errors ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { static long next = 16; *s = reinterpret_cast<cudaStream_t>(next += 16); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { if (!s) legacyPending = false; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = lastError; lastError = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return lastError; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }

// ---- the device: a B200's limits ----
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    switch (a) {
    case cudaDevAttrMultiProcessorCount: *v = sms; break;
    case cudaDevAttrMaxSharedMemoryPerBlockOptin: *v = 227 * 1024; break;
    case cudaDevAttrL2CacheSize: *v = 126 << 20; break;
    case cudaDevAttrComputeCapabilityMajor: *v = 10; break;
    case cudaDevAttrMaxGridDimX: *v = 0x7fffffff; break;
    case cudaDevAttrMaxSharedMemoryPerBlock: *v = 48 * 1024; break;
    case cudaDevAttrComputeCapabilityMinor: *v = 0; break;
    default: *v = 1;
    }
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    a->sharedSizeBytes = 2048;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    if (v + 2048 > 227 * 1024) return fail(cudaErrorInvalidValue);
    if (smemAttr.count(f) && v < smemAttr[f]) note("lowered " + names[f]);
    smemAttr[f] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int threads, size_t smem) {
    *n = (int)std::min<size_t>(2048 / threads, (228 * 1024) / (smem + 1024 + 2048));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, size_t smem, unsigned) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, threads, smem);
}
}
