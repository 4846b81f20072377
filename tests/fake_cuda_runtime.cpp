// A stand-in for the CUDA runtime, for tests of launchers on a machine without a GPU: several devices, the shared-memory attribute of a
// kernel on each, launches that are refused where the attribute is missing, and one device flag whose value a kernel still running
// leaves behind only when the device is waited for.
#include <cuda_runtime_api.h>

#include <map>
#include <utility>

namespace {
int device = 0, launches = 0, flag = 0, pending = 0, copies_fail = 0;
cudaError_t last = cudaSuccess;
std::map<std::pair<int, const void*>, int> granted;
cudaError_t launch(const void* f, size_t smem) {
    auto it = granted.find({device, f});
    if (smem > 48 * 1024 && (it == granted.end() || (size_t)it->second < smem)) return last = cudaErrorInvalidValue;
    ++launches;
    return cudaSuccess;
}
}  // namespace

extern "C" {
__attribute__((visibility("default"))) void fake_device(int d) { device = d; }
__attribute__((visibility("default"))) int fake_launches() { return launches; }
__attribute__((visibility("default"))) void fake_flag(int now, int when_waited_for, int fail) { flag = now, pending = when_waited_for, copies_fail = fail; }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static thread_local dim3 pushed[2];
static thread_local size_t pushed_smem;
static thread_local cudaStream_t pushed_stream;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    pushed[0] = grid, pushed[1] = block, pushed_smem = smem, pushed_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
    *grid = pushed[0], *block = pushed[1], *smem = pushed_smem, *(cudaStream_t*)s = pushed_stream;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int bytes) { return granted[{device, f}] = bytes, cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->dynamicSmemBytes); }
cudaError_t cudaMalloc(void** p, size_t) { return *p = nullptr, cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; return last = cudaSuccess, e; }
const char* cudaGetErrorString(cudaError_t) { return "refused by the stand-in"; }
cudaError_t cudaDeviceSynchronize() {
    if (pending) flag = pending, pending = 0;
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* dst, const void*, size_t, size_t, cudaMemcpyKind) {
    if (copies_fail) return cudaErrorUnknown;
    return *(int*)dst = flag, cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void* src, size_t, size_t, cudaMemcpyKind) { return flag = *(const int*)src, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { return *n = 0, cudaSuccess; }
static int encode_anything() { return 0; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* r) {
    return *p = (void*)encode_anything, *r = cudaDriverEntryPointSuccess, cudaSuccess;
}
}
