// A CUDA runtime for the library's host code on a machine without a GPU: device
// memory is host memory, kernels do not run, and every launch is held to the
// rules that the real runtime enforces on the host.  In particular the limit of
// a kernel's dynamic shared memory (cudaFuncAttributeMaxDynamicSharedMemorySize)
// belongs to the kernel on one device; a launch above it is refused.
// Linked with the library's objects in the place of the CUDA runtime.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

// hook(event, name, pointer, value): called before "launch" (kernel name, its
// arguments, dynamic shared memory), "occupancy" (kernel name) and after "copy"
// (direction, destination, bytes); a result other than 0 is the call's error.
typedef int (*Hook)(const char*, const char*, void*, long);

namespace {
std::mutex mu;
std::map<const void*, std::string> kernels;
std::map<std::pair<int, const void*>, int> limits;  // dynamic shared memory by device and kernel
Hook hook = nullptr;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local Config config;
constexpr int kSharedOptin = 232448, kSharedDefault = 49152;

cudaError_t fail(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
std::string name_of(const void* f) {
  std::lock_guard<std::mutex> lk(mu);
  auto it = kernels.find(f);
  return it == kernels.end() ? "?" : it->second;
}
int tell(const char* event, const char* name, void* p, long v) { return hook ? hook(event, name, p, v) : 0; }

cudaError_t launch(const void* f, dim3 grid, dim3 block, void** args, size_t smem) {
  int limit = kSharedDefault;
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = limits.find({device, f});
    if (it != limits.end()) limit = it->second;
  }
  const long refused = grid.x == 0 || grid.y == 0 || grid.z == 0 || grid.y > 65535 || grid.z > 65535 ||
                       block.x * block.y * block.z > 1024 || (long)smem > limit;
  const int told = tell(refused ? "refused" : "launch", name_of(f).c_str(), args, (long)smem);
  if (refused) return fail(cudaErrorInvalidValue);
  return fail((cudaError_t)told);
}
cudaError_t copy(void* dst, const void* src, size_t n, const char* kind) {
  if (n) std::memcpy(dst, src, n);
  return fail((cudaError_t)tell("copy", kind, dst, (long)n));
}
const char* direction(cudaMemcpyKind k) {
  return k == cudaMemcpyDeviceToHost ? "to host" : (k == cudaMemcpyHostToDevice ? "to device" : "on device");
}
CUresult encode_tiled(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
}  // namespace

extern "C" {
void fake_hook(Hook h) { hook = h; }
void fake_device(int d) { device = d; }

void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  std::lock_guard<std::mutex> lk(mu);
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* stream) {
  config = Config{grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *(cudaStream_t*)stream = config.stream;
  return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t) {
  return launch(f, grid, block, args, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return launch(f, c->gridDim, c->blockDim, args, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v > kSharedOptin) return fail(cudaErrorInvalidValue);
    std::lock_guard<std::mutex> lk(mu);
    limits[{device, f}] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t, unsigned) {
  *n = 1;
  return fail((cudaError_t)tell("occupancy", name_of(f).c_str(), nullptr, 0));
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = 8;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? kSharedOptin : 1);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  if (n) std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return copy(d, s, n, direction(k));
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, direction(k)); }
cudaError_t cudaMemcpyFromSymbolAsync(void* d, const void*, size_t n, size_t, cudaMemcpyKind, cudaStream_t) {
  std::memset(d, 0, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return fail(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return fail(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)1;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *p = (void*)encode_tiled;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}
