// Post-processing on the device, next to the solution already in HBM:
//   * centroid von Mises stress  (core/fea.py:604-626)
//   * element strain energy u_e^T KE u_e  (core/fea.py:595-602)
// and the pre-step that drops voxel islands not connected to a support
// (core/fea.py:165-227) as an in-place 6-connected flood fill.
#include "../../include/voxfea.h"
#include "vf_common.cuh"
#include "vf_workspace.cuh"

namespace vf {

namespace {

struct B0Tab { double b[6 * 24]; };
struct KETab { double k[576]; };

__device__ __forceinline__ void gather_ue(const Grid& g, const double* __restrict__ u, int ix, int iy, int iz,
                                          double ue[24]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ox = (k == 1 || k == 2 || k == 5 || k == 6);
    const int oy = (k == 2 || k == 3 || k == 6 || k == 7);
    const int oz = (k >= 4);
    const long long p = 3 * (long long)g.idx(ix + ox, iy + oy, iz + oz);
    ue[3 * k] = u[p]; ue[3 * k + 1] = u[p + 1]; ue[3 * k + 2] = u[p + 2];
  }
}

__global__ void k_von_mises(Grid g, const double* __restrict__ u, const double* __restrict__ Es,
                            const double* __restrict__ nu_ref, double nu, const uint8_t* __restrict__ active,
                            const B0Tab B, double* __restrict__ vm) {
  const long long ne = (long long)g.lx * g.ly * g.lz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
    if (active && !active[e]) { vm[e] = 0.0; continue; }
    const int iz = (int)(e % g.lz);
    const long long t = e / g.lz;
    const int iy = (int)(t % g.ly), ix = (int)(t / g.ly);
    double ue[24];
    gather_ue(g, u, ix, iy, iz, ue);
    double eps[6];
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < 24; ++j) s += B.b[r * 24 + j] * ue[j];
      eps[r] = s;
    }
    const double n = nu_ref ? nu_ref[e] : nu;
    const double c = 1.0 / ((1.0 + n) * (1.0 - 2.0 * n));
    const double gsh = c * (1.0 - 2.0 * n) / 2.0;
    const double E = Es[e];
    const double sx = E * c * ((1.0 - n) * eps[0] + n * eps[1] + n * eps[2]);
    const double sy = E * c * (n * eps[0] + (1.0 - n) * eps[1] + n * eps[2]);
    const double sz = E * c * (n * eps[0] + n * eps[1] + (1.0 - n) * eps[2]);
    const double txy = E * gsh * eps[3], tyz = E * gsh * eps[4], tzx = E * gsh * eps[5];
    const double v = 0.5 * ((sx - sy) * (sx - sy) + (sy - sz) * (sy - sz) + (sz - sx) * (sz - sx)) +
                     3.0 * (txy * txy + tyz * tyz + tzx * tzx);
    vm[e] = sqrt(v > 0.0 ? v : 0.0);
  }
}

__global__ void k_strain_energy(Grid g, const double* __restrict__ u, const uint8_t* __restrict__ active,
                                const KETab K, double* __restrict__ se) {
  const long long ne = (long long)g.lx * g.ly * g.lz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
    if (active && !active[e]) { se[e] = 0.0; continue; }
    const int iz = (int)(e % g.lz);
    const long long t = e / g.lz;
    const int iy = (int)(t % g.ly), ix = (int)(t / g.ly);
    double ue[24];
    gather_ue(g, u, ix, iy, iz, ue);
    double s = 0.0;
    for (int i = 0; i < 24; ++i) {
      double ki = 0.0;
#pragma unroll
      for (int j = 0; j < 24; ++j) ki += K.k[i * 24 + j] * ue[j];
      s += ue[i] * ki;
    }
    se[e] = s;
  }
}

// seed[e] = active[e] && an element node is fixed (fea.py:165-177)
__global__ void k_island_seed(int nx, int ny, int nz, const uint8_t* __restrict__ active,
                              const uint8_t* __restrict__ fixed_node, uint8_t* __restrict__ kept) {
  const long long ne = (long long)nx * ny * nz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
    const int iz = (int)(e % nz);
    const long long t = e / nz;
    const int iy = (int)(t % ny), ix = (int)(t / ny);
    uint8_t s = 0;
    if (active[e]) {
      for (int k = 0; k < 8 && !s; ++k) {
        const int ox = k & 1, oy = (k >> 1) & 1, oz = k >> 2;
        const long long nid = (ix + ox) + (long long)(nx + 1) * ((iy + oy) + (long long)(ny + 1) * (iz + oz));
        s = fixed_node[nid];
      }
    }
    kept[e] = s ? 1 : 0;
  }
}

// One pass of the fill (monotone: kept only grows, so any visiting order
// reaches the same fixed point as fea.py:193-204's synchronous passes).  A
// block owns a tile of voxels and dilates it in shared memory until the tile
// no longer changes, so a pass carries the fill across whole tiles: one voxel
// a pass took 104 launches and 13 host checks on a 128x96x64 part (0.9 ms).
constexpr int kFillX = 4, kFillY = 8, kFillZ = 32, kFillThreads = 256;
__global__ void __launch_bounds__(kFillThreads) k_island_grow(int nx, int ny, int nz, const uint8_t* __restrict__ active,
                                                              uint8_t* kept, int* changed) {
  constexpr int HX = kFillX + 2, HY = kFillY + 2, HZ = kFillZ + 2, PER = kFillX * kFillY * kFillZ / kFillThreads;
  __shared__ uint8_t s_kept[HX][HY][HZ];
  const int tz = (nz + kFillZ - 1) / kFillZ, ty = (ny + kFillY - 1) / kFillY;
  const int z0 = (int)(blockIdx.x % tz) * kFillZ, y0 = (int)(blockIdx.x / tz % ty) * kFillY;
  const int x0 = (int)(blockIdx.x / tz / ty) * kFillX;
  for (int i = threadIdx.x; i < HX * HY * HZ; i += kFillThreads) {
    const int iz = i % HZ, iy = i / HZ % HY, ix = i / (HZ * HY);
    const int x = x0 + ix - 1, y = y0 + iy - 1, z = z0 + iz - 1;
    const bool in = x >= 0 && x < nx && y >= 0 && y < ny && z >= 0 && z < nz;
    s_kept[ix][iy][iz] = in ? ((volatile uint8_t*)kept)[((long long)x * ny + y) * nz + z] : (uint8_t)0;
  }
  const int lz = threadIdx.x % kFillZ, ly = threadIdx.x / kFillZ;   // this thread: PER voxels along x
  const int y = y0 + ly, z = z0 + lz;
  unsigned open = 0, grown = 0;   // bit k: voxel k is active and not kept yet / became kept here
  __syncthreads();
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int x = x0 + k;
    if (x < nx && y < ny && z < nz && active[((long long)x * ny + y) * nz + z] && !s_kept[k + 1][ly + 1][lz + 1])
      open |= 1u << k;
  }
  for (;;) {
    bool any = false;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      if (!((open >> k) & 1)) continue;
      volatile uint8_t* c = &s_kept[k + 1][ly + 1][lz + 1];
      if (c[-HY * HZ] | c[HY * HZ] | c[-HZ] | c[HZ] | c[-1] | c[1]) {
        *c = 1;
        open &= ~(1u << k);
        grown |= 1u << k;
        any = true;
      }
    }
    if (!__syncthreads_or(any)) break;
  }
#pragma unroll
  for (int k = 0; k < PER; ++k)
    if ((grown >> k) & 1) ((volatile uint8_t*)kept)[((long long)(x0 + k) * ny + y) * nz + z] = 1;
  if (grown) *changed = 1;
}
static_assert(kFillY * kFillZ == kFillThreads, "one thread per column of the tile along x");

}  // namespace

void launch_von_mises(const Grid& g, const double* u_pad, const double* Es_ref, const double* nu_ref, double nu,
                      const uint8_t* active_ref, const double* B0, double* vm_ref, cudaStream_t st) {
  B0Tab B;
  for (int i = 0; i < 144; ++i) B.b[i] = B0[i];
  const long long ne = (long long)g.lx * g.ly * g.lz;
  int blocks = (int)((ne + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  launch_k(k_von_mises, blocks, 256, 0, st, g, u_pad, Es_ref, nu_ref, nu, active_ref, B, vm_ref);
}

void launch_strain_energy_tab(const Grid& g, const double* u_pad, const uint8_t* active_ref, const double* KE,
                              double* se_ref, cudaStream_t st) {
  KETab K;
  for (int i = 0; i < 576; ++i) K.k[i] = KE[i];
  const long long ne = (long long)g.lx * g.ly * g.lz;
  int blocks = (int)((ne + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  launch_k(k_strain_energy, blocks, 256, 0, st, g, u_pad, active_ref, K, se_ref);
}

// Returns the number of dilation passes run.  d_changed: one device int.
int flood_fill_islands(int nx, int ny, int nz, const uint8_t* d_active, const uint8_t* d_fixed_node,
                       uint8_t* d_kept, int* d_changed, cudaStream_t st) {
  const long long ne = (long long)nx * ny * nz;
  int blocks = (int)((ne + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  launch_k(k_island_seed, blocks, 256, 0, st, nx, ny, nz, d_active, d_fixed_node, d_kept);
  const long long tiles = ((long long)(nx + kFillX - 1) / kFillX) * ((ny + kFillY - 1) / kFillY) * ((nz + kFillZ - 1) / kFillZ);
  int passes = 0;
  const long long max_passes = 4 * ((long long)nx + ny + nz) + ne;   // monotone: ends long before
  for (;;) {
    int h_changed = 0;
    cudaMemsetAsync(d_changed, 0, sizeof(int), st);
    for (int k = 0; k < 4; ++k)
      launch_k(k_island_grow, (unsigned)tiles, kFillThreads, 0, st, nx, ny, nz, d_active, d_kept, d_changed);
    passes += 4;
    cudaMemcpyAsync(&h_changed, d_changed, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    if (!h_changed || passes > max_passes) break;
  }
  return passes;
}

}  // namespace vf

// ---------------------------------------------------------------------------
// Per-element displacement field of the result views (solve_worker.py:374-388):
// each voxel gets the mean of its 8 corner nodes' displacement magnitude.
// Reference node / element orders; host arrays in, FP32 field out.
// ---------------------------------------------------------------------------
namespace vf {
namespace {
__global__ void k_elem_disp(int nx, int ny, int nz, const double* __restrict__ u, float* __restrict__ out) {
  const long long ne = (long long)nx * ny * nz;
  const int nx1 = nx + 1, ny1 = ny + 1;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < ne; e += (long long)gridDim.x * blockDim.x) {
    const int iz = (int)(e % nz), iy = (int)((e / nz) % ny), ix = (int)(e / ((long long)nz * ny));
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {   // corner order of build_edof (fea.py:33-36)
      const int ox = (k == 1 || k == 2 || k == 5 || k == 6), oy = (k == 2 || k == 3 || k == 6 || k == 7), oz = k >= 4;
      const long long n = (ix + ox) + (long long)nx1 * ((iy + oy) + (long long)ny1 * (iz + oz));
      const double a = u[3 * n], b = u[3 * n + 1], c = u[3 * n + 2];
      s += sqrt(a * a + b * b + c * c);
    }
    out[e] = (float)(s / 8.0);
  }
}
}  // namespace
}  // namespace vf

extern "C" int vf_element_displacement(int32_t nx, int32_t ny, int32_t nz, const double* u, float* disp_out) {
  if (nx < 1 || ny < 1 || nz < 1 || !u || !disp_out) return VF_ERR_ARG;
  const size_t ndof = 3 * (size_t)(nx + 1) * (ny + 1) * (nz + 1), ne = (size_t)nx * ny * nz;
  vf::Workspace ws;
  if (!ws.open()) return VF_ERR_CUDA;
  cudaStream_t st = ws.st;
  double* d_u = nullptr;
  float* d_o = nullptr;
  if (!ws.alloc(&d_u, ndof) || !ws.alloc(&d_o, ne)) return VF_ERR_NOMEM;
  cudaMemcpyAsync(d_u, u, sizeof(double) * ndof, cudaMemcpyHostToDevice, st);
  const long long b = ((long long)ne + 255) / 256;
  vf::launch_k(vf::k_elem_disp, (int)(b < 148 * 16 ? b : 148 * 16), 256, 0, st, nx, ny, nz, (const double*)d_u, d_o);
  cudaMemcpyAsync(disp_out, d_o, sizeof(float) * ne, cudaMemcpyDeviceToHost, st);
  return cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess ? VF_ERR_CUDA : VF_OK;
}
