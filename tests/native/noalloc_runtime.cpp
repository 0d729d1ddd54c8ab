// A stand-in for the CUDA runtime: what iwpp_reconstruct_noalloc and the
// engine's host side call, with a record of the kernels loaded and launched
// and counters that "the device" reports as told.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <set>
#include <vector>

static std::set<const void*> g_loaded;
static std::vector<const void*> g_launched;
static std::vector<unsigned char> g_memory(8u << 20);
static size_t g_error_at = 0, g_ctrl_bytes = 0;
static unsigned g_error = 0;

extern "C" {
// ---- for the test
size_t engine_ctrl_bytes();
size_t engine_ctrl_error_at();
void fake_reset(unsigned error) {
    g_launched.clear();
    g_error = error;
    g_error_at = engine_ctrl_error_at();
    g_ctrl_bytes = engine_ctrl_bytes();
}
int fake_launches() { return (int)g_launched.size(); }
int fake_distinct_kernels() { return (int)std::set<const void*>(g_launched.begin(), g_launched.end()).size(); }
// engine launches of kernels that were not loaded when they were launched;
// they are from then on
int fake_launches_that_load = 0;

// ---- the runtime
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    *p = g_memory.data();
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* fn) {
    *a = cudaFuncAttributes{};
    g_loaded.insert(fn);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* fn, int, size_t, unsigned) {
    *n = 3;
    g_loaded.insert(fn);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* fn, void**) {
    if (!g_loaded.count(fn)) ++fake_launches_that_load;
    g_loaded.insert(fn);
    g_launched.push_back(fn);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void*, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memset(dst, 0, n);
    if (n == g_ctrl_bytes) std::memcpy(static_cast<unsigned char*>(dst) + g_error_at, &g_error, sizeof(g_error));
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
// kernels that are loaded right now
int fake_loaded() { return (int)g_loaded.size(); }

// ---- what compiled CUDA sources call when they are loaded and at <<< >>>
void** __cudaRegisterFatBinary(void*) { return static_cast<void**>(std::malloc(8)); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void** h) { std::free(h); }
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(fn));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
}
