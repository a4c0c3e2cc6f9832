// A CUDA runtime on the host for tests of what the library launches: device
// memory is host memory, kernels do not run, launches are recorded and handed
// to on_launch, which may write what the kernel would.  Like the real runtime
// it refuses a launch with more dynamic shared memory than its function allows.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

struct Launch {
  std::string name;  // mangled
  unsigned blocks, threads;
  size_t smem;
  bool cooperative;
};
inline std::vector<Launch> launches;
inline std::map<const void *, std::string> names;
inline std::map<const void *, size_t> allowed;  // opted-in dynamic shared memory
inline std::function<void(const Launch &, void **)> on_launch;
inline std::function<void(const void *)> on_attribute;  // after a function's attribute was set

static cudaError_t launch(const void *f, dim3 g, dim3 b, void **args, size_t smem, bool coop) {
  const size_t limit = allowed.count(f) ? allowed[f] : 48 * 1024;
  if (smem > limit) return cudaErrorInvalidValue;
  launches.push_back({names[f], g.x * g.y * g.z, b.x * b.y * b.z, smem, coop});
  if (on_launch) on_launch(launches.back(), args);
  return cudaSuccess;
}

static struct Pushed {
  dim3 g, b;
  size_t smem;
  cudaStream_t s;
} pushed;

extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *,
                            uint3 *, dim3 *, dim3 *, int *) {
  names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  pushed = {g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = pushed.g;
  *b = pushed.b;
  *smem = pushed.smem;
  *(cudaStream_t *)s = pushed.s;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t) {
  return launch(f, g, b, args, smem, false);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem,
                                        cudaStream_t) {
  return launch(f, g, b, args, smem, true);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  return launch(f, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, false);
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) allowed[f] = (size_t)v;
  if (on_attribute) on_attribute(f);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
  *n = 8;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                   unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return cudaErrorUnknown; }
cudaError_t cudaPeekAtLastError(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemset(void *p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}

#define CHECK(x)                                                   \
  do {                                                             \
    if (!(x)) {                                                    \
      std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x);          \
      std::exit(1);                                                \
    }                                                              \
  } while (0)
