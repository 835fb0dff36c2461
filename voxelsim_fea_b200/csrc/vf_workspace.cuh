// Device buffers of one call of the stateless entry points (voxelization, grid
// assembly, island removal, displacement field).
//
// cudaMalloc / cudaFree per call cost these entry points more than their
// kernels (the displacement field of a 64x32x32 grid: up to 10 ms a call, and cudaFree
// waits for every stream of the device; job on 128x64x64 67 -> 51 ms, voxel
// phase on 128x96x64 41 -> 30 ms).  The buffers come from one
// stream-ordered memory pool per device instead: it keeps at most
// kPoolKeepBytes between calls, is safe for any number of threads and streams
// (the allocator orders reuse itself), and workspace_trim gives what it keeps
// back -- every other device allocation of the library (device_malloc) does
// that before it gives up.
#pragma once

#include <cuda_runtime.h>

#include <vector>

namespace vf {

constexpr size_t kPoolKeepBytes = (size_t)512 << 20;

// The current device's pool; nullptr where the device has none.
cudaMemPool_t workspace_pool();
// Gives the pool's unused memory on the current device back.
void workspace_trim();
// cudaMalloc that, out of memory, first takes back what the pool keeps.
cudaError_t device_malloc(void** p, size_t bytes);

struct Workspace {
  std::vector<void*> p;
  cudaStream_t st = nullptr;
  cudaMemPool_t pool = nullptr;

  // false: no stream
  bool open() {
    pool = workspace_pool();
    return cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess;
  }
  template <typename T> bool alloc(T** out, size_t count) {
    const size_t bytes = count * sizeof(T) + 16;
    void* q = nullptr;
    for (int attempt = 0; attempt < 2; ++attempt) {
      const cudaError_t e = pool ? cudaMallocFromPoolAsync(&q, bytes, pool, st) : device_malloc(&q, bytes);
      if (e == cudaSuccess) {
        p.push_back(q);
        *out = (T*)q;
        return true;
      }
      cudaGetLastError();
      workspace_trim();
    }
    return false;
  }
  ~Workspace() {
    for (void* q : p) {
      if (pool) cudaFreeAsync(q, st);
      else cudaFree(q);
    }
    if (st) {
      cudaStreamSynchronize(st);
      cudaStreamDestroy(st);
    }
  }
  Workspace() = default;
  Workspace(const Workspace&) = delete;
  Workspace& operator=(const Workspace&) = delete;
};

}  // namespace vf
