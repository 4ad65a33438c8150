// Stands in for the CUDA runtime calls by which the host code of the kernel library prepares and issues launches, so that it
// runs without a GPU: devices with shared-memory limits of their own per kernel, as the runtime keeps them. Preloaded.
#include <cuda_runtime_api.h>

#include <map>
#include <mutex>
#include <utility>

namespace {
std::mutex mu;
int device = 0, clusters[8] = {40, 40, 40, 40, 40, 40, 40, 40}, last_grid_x = 0, launches = 0;
cudaError_t last_error = cudaSuccess;
std::map<std::pair<int, const void*>, int> limit;   // dynamic shared memory that a kernel may have on a device; 48 KB with the static one unasked

cudaError_t launch(const void* f, unsigned grid_x, size_t smem) {
  std::lock_guard<std::mutex> l(mu);
  const auto it = limit.find({device, f});
  if (smem > (size_t)(it == limit.end() ? 47 * 1024 : it->second)) return last_error = cudaErrorInvalidValue;
  last_grid_x = (int)grid_x;
  ++launches;
  return cudaSuccess;
}
int encode(...) { return 0; }   // cuTensorMapEncodeTiled
}  // namespace

extern "C" {
void fake_set_device(int d) { device = d; }
void fake_set_clusters(int d, int n) { clusters[d] = n; }
int fake_last_grid_x() { return last_grid_x; }
int fake_launches() { return launches; }

cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> l(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) limit[{device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = clusters[device];
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim.x, c->dynamicSmemBytes);
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void**, size_t smem, cudaStream_t) {
  return launch(f, grid.x, smem);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *f = (void*)encode;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}
