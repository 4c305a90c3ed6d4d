// TEST ONLY: the CUDA runtime calls of the engine over two pretended devices,
// so that the host code around the kernels can run where no GPU is.  Device
// memory is host memory, kernels do nothing, events take no time.  Calls that
// act on the current device are counted when that is not the device the test
// expects (fake_expect).  Linked with the engine's objects in place of the
// runtime by tests/native/build.py; never part of the product.
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdlib>
#include <cstring>

namespace {
thread_local int current = 0;
std::atomic<int> expected{0}, wrong{0}, launches{0};
int here() {
  if (current != expected) ++wrong;
  return current;
}
template <class T>
cudaError_t handle(T *out) {
  static std::atomic<uintptr_t> next{4096};
  *out = reinterpret_cast<T>(next += 16);
  return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_expect(int device) {
  expected = device;
  wrong = launches = 0;
}
int fake_wrong() { return wrong; }
int fake_launches() { return launches; }

cudaError_t cudaGetDeviceCount(int *n) { return *n = 2, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = current, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return current = d, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 1;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = size_t(1) << 37, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
const char *cudaGetErrorName(cudaError_t) { return "fake"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  static double array[1 << 16];
  return *p = array, cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *, void **, unsigned long long, cudaDriverEntryPointQueryResult *) {
  return cudaErrorNotSupported;
}

cudaError_t cudaMalloc(void **p, size_t n) { return here(), *p = std::calloc(1, n ? n : 1), cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = std::calloc(1, n ? n : 1), cudaSuccess; }
cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return std::free(p), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return std::memmove(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return std::memmove(d, s, n), cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }

cudaError_t cudaEventCreate(cudaEvent_t *e) { return here(), handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return here(), handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreate(cudaStream_t *s) { return here(), handle(s); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return here(), handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { return here(), handle(e); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

cudaError_t cudaLibraryLoadData(cudaLibrary_t *l, const void *, cudaJitOption *, void **, unsigned,
                                cudaLibraryOption *, void **, unsigned) {
  return handle(l);
}
cudaError_t cudaLibraryGetKernel(cudaKernel_t *k, cudaLibrary_t, const char *) { return handle(k); }
cudaError_t cudaLibraryUnload(cudaLibrary_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return here(), cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
  return here(), *n = 2, cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) {
  return here(), ++launches, cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  *g = *b = dim3(1, 1, 1);
  *s = 0;
  *static_cast<cudaStream_t *>(st) = nullptr;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
  static void *h[1];
  return h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
