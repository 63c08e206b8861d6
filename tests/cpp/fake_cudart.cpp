// A CUDA runtime for tests without a GPU: device memory is host memory, kernels do nothing but leave
// their names in a list, and a call can be made to fail.  Linked with the engine's objects in place of
// the CUDA runtime, it shows what the engine's host code does after an error.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

#include "rp_internal.cuh"

namespace {

std::map<const void *, std::string> names;
std::string launched;
std::string fail_call;
int fail_after = -1;
int allocations = 0;
rp::SoftSweepArgs soft{};   // of the last FP64 sweep
cudaError_t last_error = cudaSuccess;
struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} config;

// The error of a call that is to fail: the `fail_after`th from now on of that name.
bool fails(const char *call) {
    if (fail_after < 0 || fail_call != call) return false;
    return fail_after-- == 0;
}

cudaError_t allocate(const char *call, void **p, size_t bytes) {
    *p = nullptr;
    if (fails(call)) return cudaErrorMemoryAllocation;
    *p = std::calloc(1, bytes ? bytes : 1);
    allocations++;
    return cudaSuccess;
}

cudaError_t launch(const void *f, void **args) {
    const auto it = names.find(f);
    const std::string name = it == names.end() ? "?" : it->second;
    if (fails("launch") || (fail_after >= 0 && name.find(fail_call) != std::string::npos && fail_after-- == 0))
        return last_error = cudaErrorLaunchOutOfResources;
    launched += name + "\n";
    if (name.find("k_soft_sweep") != std::string::npos) soft = *static_cast<const rp::SoftSweepArgs *>(args[0]);
    return cudaSuccess;
}

}  // namespace

extern "C" {

// The `after`th next call of `call` (a runtime function's name, or a part of a kernel's) fails.
void fake_fail(const char *call, int after) {
    fail_call = call;
    fail_after = after;
}
// The kernels launched since the last call, one a line.
const char *fake_launched() {
    static std::string out;
    out.swap(launched);
    launched.clear();
    return out.c_str();
}
// The allocations since the last call that did not fail.
int fake_allocations() {
    const int n = allocations;
    allocations = 0;
    return n;
}

// Whether the last FP64 sweep was to do without the FP32 filter.
int fake_soft_fp64_only() { return soft.c.fp64_only; }

void **__cudaRegisterFatBinary(void *) {
    static void *handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *device, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    names[host] = device;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, CUstream_st *stream) {
    config = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *static_cast<cudaStream_t *>(stream) = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **args, size_t, cudaStream_t) { return launch(k, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *f, void **args) { return launch(f, args); }

cudaError_t cudaMalloc(void **p, size_t bytes) { return allocate("cudaMalloc", p, bytes); }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return allocate("cudaHostAlloc", p, bytes); }
cudaError_t cudaFree(void *p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void *to, const void *from, size_t n, cudaMemcpyKind) {
    if (fails("cudaMemcpy")) return cudaErrorUnknown;
    std::memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fails("cudaMemcpyAsync")) return cudaErrorUnknown;
    std::memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
    if (fails("cudaMemsetAsync")) return cudaErrorUnknown;
    return cudaMemset(p, v, n);
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 227 * 1024;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetLimit(size_t *v, cudaLimit) {
    *v = 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    *a = cudaPointerAttributes{};
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *s) {
    *p = const_cast<void *>(s);
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "a fake error"; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
}
