// A CUDA runtime of two devices that launches nothing, for the launchers' host code: it keeps which kernel
// may use how much dynamic shared memory on which device, refuses launches that ask for more, and refuses
// what a stream capture refuses.  Linked with the kernels' objects in place of the real runtime.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <map>
#include <utility>

namespace {
int64_t last_threads = 0;
int device = 0, launches = 0, capturing = 0, refused_in_capture = 0;
cudaError_t last = cudaSuccess;
std::map<std::pair<int, const void*>, int> smem_limit;
int words[2];                                          // a device variable, one for each device

cudaError_t keep(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t not_in_capture() {
  if (!capturing) return cudaSuccess;
  refused_in_capture++;
  return keep(cudaErrorStreamCaptureUnsupported);
}
cudaError_t launch(const void* kern, size_t smem, dim3 grid, dim3 block) {
  auto it = smem_limit.find({device, kern});
  if (smem > (size_t)(it == smem_limit.end() ? 48 * 1024 : it->second)) return keep(cudaErrorInvalidValue);
  launches++;
  last_threads = (int64_t)grid.x * grid.y * grid.z * block.x * block.y * block.z;
  return cudaSuccess;
}
CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
}  // namespace

extern "C" {
// for the tests
void host_use_device(int dev) { device = dev; }
void host_capture(int on) { capturing = on; refused_in_capture = 0; }
int host_refused_in_capture() { return refused_in_capture; }
int host_launches() { return launches; }
int64_t host_last_threads() { return last_threads; }
void ft_note_launches(int) {}

// the runtime
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) { *p = &words[device]; return not_in_capture(); }
cudaError_t cudaFree(void* p) { return p ? not_in_capture() : cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return not_in_capture(); }
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return not_in_capture(); }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = &words[device]; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_limit[{device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
  return launch(f, smem, grid, block);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->dynamicSmemBytes, c->gridDim, c->blockDim);
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *p = (void*)encode;
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
