// A CUDA runtime without a GPU, linked in place of the real one with the library's
// own objects: launches and copies are written down, memory is address space, and
// an allocation can be made to fail.  Host logic of the launchers and the C
// interface runs on it as it is.
#include <sys/mman.h>

#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

#include "launch.h"

namespace {
std::mutex mu;
std::map<const void*, std::string> kernels;  // by host stub
std::map<uintptr_t, size_t> blocks;          // device memory
std::string log_text;
uint64_t live = 0, peak = 0, allocations = 0;
int fail_at = 0, device = 0, per_sm = 4;
std::vector<int> sms(64, 148);
cudaError_t last = cudaSuccess;
struct Config { dim3 grid, block; size_t shmem; cudaStream_t s; };
thread_local std::vector<Config> configs;

cudaError_t result(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
cudaError_t allocate(void** p, size_t n) {
    std::lock_guard<std::mutex> lock(mu);
    *p = nullptr;
    allocations++;
    if (fail_at > 0 && --fail_at == 0) return result(cudaErrorMemoryAllocation);
    void* m = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return result(cudaErrorMemoryAllocation);
    blocks[(uintptr_t)m] = n ? n : 1;
    live += n;
    if (live > peak) peak = live;
    *p = m;
    return cudaSuccess;
}
cudaError_t release(void* p) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = blocks.find((uintptr_t)p);
    if (it == blocks.end()) return result(p ? cudaErrorInvalidValue : cudaSuccess);
    live -= it->second;
    munmap(p, it->second);
    blocks.erase(it);
    return cudaSuccess;
}
bool on_device(const void* p) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = blocks.upper_bound((uintptr_t)p);
    if (it == blocks.begin()) return false;
    --it;
    return (uintptr_t)p < it->first + it->second;
}
void note(const std::string& s) {
    std::lock_guard<std::mutex> lock(mu);
    log_text += s + "\n";
}
}  // namespace

extern "C" {
// ------------------------------------------------------------- the runtime
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shmem, cudaStream_t s) {
    configs.push_back({grid, block, shmem, s});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shmem, void* s) {
    const Config c = configs.back();
    configs.pop_back();
    *grid = c.grid, *block = c.block, *shmem = c.shmem;
    *static_cast<cudaStream_t*>(s) = c.s;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t, cudaStream_t) {
    note("launch " + kernels[f] + " " + std::to_string(grid.x) + " " + std::to_string(block.x));
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return allocate(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return release(p); }
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaMemcpyAsync(void* d, const void*, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    if (kind == cudaMemcpyDeviceToHost) memset(d, 0, n);
    if (kind == cudaMemcpyDeviceToDevice)
        note("copy " + std::to_string((uintptr_t)d) + " " + std::to_string(n));
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void*, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    if (w > dp || w > sp) return result(cudaErrorInvalidPitchValue);
    for (size_t i = 0; i < h; i++) note("copy " + std::to_string((uintptr_t)d + i * dp) + " " + std::to_string(w));
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    memset(a, 0, sizeof(*a));
    a->type = on_device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    a->device = device;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) {
    *p = const_cast<void*>(symbol);  // part of the image, not allocated
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int dev) {
    *v = a == cudaDevAttrMultiProcessorCount ? sms[dev] : 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = per_sm;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    device = d;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 64;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    *f = *t = size_t(180) << 30;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1;
    return cudaSuccess;
}

// ----------------------------------------------------------- for the tests
void fake_fail_at(int n) { fail_at = n; }
void fake_per_sm(int n) { per_sm = n; }
void fake_device(int d, int count) { device = d, sms[d] = count; }
uint64_t fake_live() { return live; }
uint64_t fake_allocations() { return allocations; }
uint64_t fake_peak() {
    const uint64_t p = peak;
    peak = live;
    return p;
}
// what was launched and copied since the last call
const char* fake_log() {
    static std::string text;
    text.swap(log_text);
    log_text.clear();
    return text.c_str();
}
void* fake_buffer(uint64_t n) {
    void* p = nullptr;
    allocate(&p, n);
    return p;
}
void fake_free(void* p) { release(p); }
int fake_error() { return (int)cudaGetLastError(); }

using namespace wbte;
static uint8_t* const ANY = reinterpret_cast<uint8_t*>(uintptr_t(1) << 40);
int h_miller_lines_multi(int64_t n, int64_t per, int64_t T) {
    return launch_miller_lines_multi(ANY, ANY, ANY, n, per, (int)T, nullptr);
}
// window, segments per window and scratch of a plan (the window 0: none within `limit`)
void h_msm_plan(int g, int64_t n, int64_t k, uint64_t limit, int64_t* out) {
    const MsmPlan p = msm_plan((Group)g, n, k, limit ? limit : SIZE_MAX);
    out[0] = p.c, out[1] = p.segments, out[2] = p.c ? (int64_t)msm_family_scratch_bytes((Group)g, 1, k, n, p) : 0;
}
void h_fp12_mul(int64_t n) { launch_fp12_mul(ANY, ANY, 1, ANY, 1, false, n, nullptr); }
}
