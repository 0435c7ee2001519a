// A stand-in for the CUDA runtime, for tests of the library's host code without a GPU: memory is the
// host's, launches run nothing, and the next launch of a named kernel can be made to fail.  It follows
// the one thing those tests ask about, the host array that the step's descriptor points at.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void*, std::string>& names() {  // kernels are registered before this file's own globals exist
  static std::map<const void*, std::string> m;
  return m;
}
std::string failing;
char handle;  // what streams, events and graphs point at
cudaError_t last = cudaSuccess;
void* host_u = nullptr;
struct Call {
  dim3 grid, block;
  size_t smem;
  cudaStream_t s;
} pending;

cudaError_t run(const void* fun, void** args) {
  const std::string& name = names()[fun];
  if (!failing.empty() && name.find(failing) != std::string::npos) {
    failing.clear();
    return last = cudaErrorLaunchOutOfResources;
  }
  if (name.find("k_open_run") != std::string::npos && *(void**)args[1]) host_u = *(void**)args[2];
  if (name.find("k_set_host_u") != std::string::npos) host_u = *(void**)args[1];
  return cudaSuccess;
}
int encode_tiled(...) { return 0; }
}  // namespace

extern "C" {
void fake_reset(const char* kernel) {  // the next launch of a kernel of this name (none if empty) fails
  failing = kernel;
  host_u = nullptr;
}
void* fake_host_u() { return host_u; }

void** __cudaRegisterFatBinary(void*) { return (void**)&handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* fun, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names()[fun] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  pending = Call{g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = pending.grid;
  *b = pending.block;
  *smem = pending.smem;
  *(cudaStream_t*)s = pending.s;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fun) {
  *k = (cudaKernel_t)fun;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t, cudaStream_t) { return run((const void*)k, args); }
cudaError_t cudaLaunchKernel(const void* fun, dim3, dim3, void** args, size_t, cudaStream_t) { return run(fun, args); }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the stand-in"; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceCanAccessPeer(int* v, int, int) { *v = 0; return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned) { return cudaErrorPeerAccessUnsupported; }
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
  for (size_t r = 0; r < h; r++) memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {  // every array is page-locked and mapped
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeHost;
  a->devicePointer = a->hostPointer = const_cast<void*>(p);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *p = (void*)encode_tiled;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)&handle; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)&handle; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)&handle; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)&handle; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 1.0f; return cudaSuccess; }
}
