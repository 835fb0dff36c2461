// The device memory pools behind Workspace (vf_workspace.cuh).
#include "vf_workspace.cuh"

#include <mutex>

#include "vf_common.cuh"

namespace vf {

namespace {
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};
bool g_tried[kMaxDevices] = {};
}  // namespace

cudaMemPool_t workspace_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_tried[dev]) {
    g_tried[dev] = true;
    int ok = 0;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && ok &&
        cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
      unsigned long long keep = kPoolKeepBytes;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
      g_pool[dev] = pool;
    }
    cudaGetLastError();
  }
  return g_pool[dev];
}

void workspace_trim() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (g_pool[dev]) cudaMemPoolTrimTo(g_pool[dev], 0);
  cudaGetLastError();
}

cudaError_t device_malloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    workspace_trim();
    e = cudaMalloc(p, bytes);
  }
  return e;
}

}  // namespace vf
