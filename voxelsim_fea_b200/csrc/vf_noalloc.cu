// vf_apply_noalloc: the fine-level hex8 operator y = mask(K u) with the fused
// dot product u.y, for callers that cannot allocate device memory.
//
// Who needs it: an application that owns every byte of device memory through
// its own allocator or a fixed arena (a solver embedded in a larger program
// with a hard memory budget), and code that must not trigger the implicit
// device synchronisation cudaMalloc/cudaFree can cause (real-time loops,
// work issued between other streams' kernels).  Such a caller passes its own
// device buffers; this entry point creates no solver handle and calls no
// allocator.  The only scratch -- one FP64 partial sum per thread block and a
// completion counter for the dot product -- lives in the fixed array below,
// which every GPU that loads the library keeps until the process exits.
//
// Limits and sharing:
//   * at most kMaxBlocks blocks of 256 threads, i.e. (nx+1)(ny+1)(nz+1) <=
//     kMaxNodes grid nodes; larger grids are rejected with VF_ERR_ARG;
//   * every call on a device shares the one array and it keeps the last call's
//     contents; successive calls on a device take successive completion
//     counters of a ring, and a call's last block clears its own and the one
//     half a ring ahead, so a counter that an overlap spoilt does not stay
//     spoilt.  A captured call would keep its counter for every replay: it
//     takes one outside the ring, cleared by a memset node ahead of the kernel;
//     Calls whose kernels overlap on the GPU (different streams, no ordering)
//     race on the array and give wrong results: order them on one stream;
//   * the first call on each device looks up the array's device address
//     (cudaGetSymbolAddress with that device current), keeps it for the
//     process and loads both forms' kernels; make that first call, on any
//     grid, before any stream capture.  A
//     cudaDeviceReset tears the module down with the context, so the kept
//     address is stale afterwards: make no call on that device after a reset;
//   * u, y and u_dot_y must not overlap: threads read u at neighbouring nodes
//     while others write y, so an in-place call is rejected.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>

#include "../../include/voxfea.h"
#include "vf_common.cuh"
#include "vf_hex8.h"
#include "vf_modal.cuh"

namespace vf {
extern thread_local std::string g_last_error;
}

namespace {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 32768;
constexpr long long kMaxNodes = (long long)kMaxBlocks * kThreads;   // 8,388,608 nodes
constexpr int kMaxDevices = 64;
constexpr int kRing = 64;
// [0, kMaxBlocks) doubles: per-block partials; then the ring's counters and the captured calls'.
constexpr size_t kScratchBytes = sizeof(double) * kMaxBlocks + (kRing + 1) * sizeof(unsigned);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

struct KeParam { double k[576]; };

unsigned char* g_scratch_addr[kMaxDevices] = {};
std::mutex g_scratch_mu;
std::atomic<unsigned> g_call[kMaxDevices];
std::atomic<int> g_march_ready[vf::kMaxDevices];

// Block sum in a fixed order; the last block sums the partials in order.
__device__ __forceinline__ void finish_dot(double dot, double* __restrict__ dot_out, double* __restrict__ partials,
                                           unsigned int* __restrict__ counters, unsigned slot, unsigned heal) {
  __shared__ double s_w[kThreads / 32];
  __shared__ bool s_last;
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if ((tid & 31) == 0) s_w[tid >> 5] = dot;
  __syncthreads();
  if (tid == 0) {
    double b = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) b += s_w[w];
    partials[blockIdx.x] = b;
    __threadfence();
    s_last = (atomicAdd(counters + slot, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double s = 0.0;
  for (int i = tid; i < (int)gridDim.x; i += kThreads) s += ((volatile double*)partials)[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((tid & 31) == 0) s_w[tid >> 5] = s;
  __syncthreads();
  if (tid == 0) {
    double tot = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) tot += s_w[w];
    *dot_out = tot;
    counters[slot] = 0u;
    counters[heal] = 0u;
  }
}

// The operator in modal form (vf_modal.cuh), marching along z: 32 x 8 threads
// own a 31 x 7 tile of nodes and a chunk of planes; each thread transforms the
// face of its element column once per plane, couples it with the plane below
// and keeps the upper face's forces for the next step, so a node's value is
// loaded once per tile and a voxel costs ~170 operations instead of the 576
// products per node of the gather form below.  The caller's arrays are in
// reference order with rows of any alignment, so planes are staged with
// 8-byte asynchronous copies, two planes ahead in a ring of four (staged
// through registers they cost spills and waits: 161 us where it is 118 now);
// the corner forces are exchanged through a double buffer, one barrier a
// plane.  Bound by the FP64 and shared-memory instructions of 16 warps an SM
// (the 24 modes of a voxel and their forces fill the registers).  251x127x129
// voxels: 387 us (gather) -> 117 us; 48x24x24: 29 -> 9.3 us (there also without a
// clearing launch and the host's 24x24 tables).
constexpr int kMX = 32, kMY = 8;
constexpr int kRow = 3 * (kMX + 1), kPlane = (kMY + 1) * kRow;   // 33 x 9 halo nodes
constexpr size_t kMarchSmem = sizeof(double) * (4 * kPlane + 2 * 3 * 3 * kMY * kMX);
struct March { int ntx, nty, zchunk; long long units, steps; };

// 8-byte asynchronous copy to shared memory; zeros where !in
__device__ __forceinline__ void copy8(double* dst, const double* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__global__ void __launch_bounds__(kThreads, 2)
    k_apply_march(int nx, int ny, int nz, const double* __restrict__ E, const uint8_t* __restrict__ mask,
                  const double* __restrict__ u, double* __restrict__ y, double* __restrict__ dot_out,
                  double* __restrict__ partials, unsigned int* __restrict__ counters, unsigned slot, unsigned heal,
                  const vf::ModalConst mc, March mp) {
  using O = vf::modal::Pack<double>;
  extern __shared__ double smem[];
  double (*s_u)[kPlane] = reinterpret_cast<double (*)[kPlane]>(smem);
  double (*s_c)[3][3][kMY][kMX] = reinterpret_cast<double (*)[3][3][kMY][kMX]>(smem + 4 * kPlane);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + kMX * ty;
  const int nx1 = nx + 1, ny1 = ny + 1;
  constexpr int NL = (3 * (kMX + 1) * (kMY + 1) + kThreads - 1) / kThreads;   // halo values per thread
  double dot = 0.0;
  const int unit = blockIdx.x;
  const int X0 = unit % mp.ntx * (kMX - 1), Y0 = unit / mp.ntx % mp.nty * (kMY - 1);
  const int zb = unit / (mp.ntx * mp.nty) * mp.zchunk, ze = min(zb + mp.zchunk, nz + 1);
  const int Xc = X0 - 1 + tx, Yc = Y0 - 1 + ty;
  const bool out_col = tx >= 1 && ty >= 1 && Xc <= nx && Yc <= ny;
  const bool elem_col = Xc >= 0 && Xc < nx && Yc >= 0 && Yc < ny;
  const double* Ecol = E + (elem_col ? ((long long)Xc * ny + Yc) * nz : 0);
  const int node_col = out_col ? Xc + nx1 * Yc : 0;
  int goff[NL];   // this thread's halo values tid + q * kThreads: offset within a plane of u (-1: outside)
#pragma unroll
  for (int q = 0; q < NL; ++q) {
    const int e = tid + q * kThreads, j = e / kRow, i = e % kRow;
    const int gx = X0 - 1 + i / 3, gy = Y0 - 1 + j;
    goff[q] = (j < kMY + 1 && gx >= 0 && gx <= nx && gy >= 0 && gy <= ny) ? 3 * (gx + nx1 * gy) + i % 3 : -1;
  }
  auto fetch = [&](int z, int b) {
    const bool zin = z >= 0 && z <= nz;
    const double* up = u + (zin ? 3LL * nx1 * ny1 * z : 0);
#pragma unroll
    for (int q = 0; q < NL; ++q)
      if (tid + q * kThreads < kPlane) copy8(&s_u[b][tid + q * kThreads], up + max(goff[q], 0), zin && goff[q] >= 0);
  };
  double hiPrev[3][4], Fp[3][4];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int m = 0; m < 4; ++m) { hiPrev[c][m] = 0.0; Fp[c][m] = 0.0; }
  // plane s of this unit is z = zb - 1 + s; layer s lies between planes s - 1 and s
  const int nsteps = ze - zb + 2;
  fetch(zb - 1, 0);
  copy_commit();
  fetch(zb, 1);
  copy_commit();
  double En = 0.0;
  uint8_t mk = 0;
  copy_wait1();
  __syncthreads();
#pragma unroll 1
  for (int s = 0; s < nsteps; ++s) {
    const int z = zb - 1 + s;
    // (slot (s + 2) & 3 was last read before the barrier of step s - 1)
    if (s + 2 < nsteps) fetch(z + 2, (s + 2) & 3);
    copy_commit();
    const double Ee = En;   // of layer s
    En = (elem_col && z >= 0 && z < nz && s + 1 < nsteps) ? __ldg(Ecol + z) : 0.0;
    const uint8_t m8 = mk;
    mk = (out_col && s >= 1 && z >= 0 && z <= nz) ? __ldg(mask + node_col + (long long)nx1 * ny1 * z) : (uint8_t)0;
    const double* us = s_u[s & 3] + ty * kRow + 3 * tx;
    double Fc[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double u00 = us[c], u10 = us[3 + c], u01 = us[kRow + c], u11 = us[kRow + 3 + c];
      const double e0 = u10 + u00, e1 = u10 - u00, e2 = u11 + u01, e3 = u11 - u01;
      Fc[c][0] = e0 + e2;
      Fc[c][1] = e1 + e3;
      Fc[c][2] = e2 - e0;
      Fc[c][3] = e3 - e1;
    }
    if (s >= 1) {
      double A[3][8], B[3][8];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          A[c][m] = Fp[c][m] + Fc[c][m];
          A[c][m + 4] = Fc[c][m] - Fp[c][m];
        }
      vf::modal::modal_physics<O, double, double>(A, B, Ee, Ee, mc);
      double c00[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double acc[4];
        acc[0] = hiPrev[c][0] - B[c][4];
        hiPrev[c][0] = B[c][4];
#pragma unroll
        for (int m = 1; m < 4; ++m) {
          acc[m] = hiPrev[c][m] + (B[c][m] - B[c][m + 4]);
          hiPrev[c][m] = B[c][m] + B[c][m + 4];
        }
        const double t0 = acc[0] - acc[2], t1 = acc[1] - acc[3], t2 = acc[0] + acc[2], t3 = acc[1] + acc[3];
        c00[c] = t0 - t1;
        s_c[s & 1][0][c][ty][tx] = t0 + t1;
        s_c[s & 1][1][c][ty][tx] = t2 - t3;
        s_c[s & 1][2][c][ty][tx] = t2 + t3;
      }
      double own[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) own[c] = s_u[(s - 1) & 3][ty * kRow + 3 * tx + c];
      copy_wait1();   // plane s + 1 of this thread; the barrier makes it all threads'
      __syncthreads();
      if (s >= 2 && out_col) {
        const long long p3 = 3 * (node_col + (long long)nx1 * ny1 * (z - 1));
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double v = (c00[c] + s_c[s & 1][0][c][ty][tx - 1]) +
                           (s_c[s & 1][1][c][ty - 1][tx] + s_c[s & 1][2][c][ty - 1][tx - 1]);
          const double k = ((m8 >> c) & 1) ? v : 0.0;
          y[p3 + c] = k;
          dot += own[c] * k;
        }
      }
    } else {
      copy_wait1();
      __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int m = 0; m < 4; ++m) Fp[c][m] = Fc[c][m];
  }
  finish_dot(dot, dot_out, partials, counters, slot, heal);
}

// The operator as a node-centric gather over KE, one thread per node: better
// on grids too thin to fill the marching form's tiles.
__global__ void __launch_bounds__(kThreads) k_apply_noalloc(int nx, int ny, int nz, const double* __restrict__ E,
                                                            const uint8_t* __restrict__ mask,
                                                            const double* __restrict__ u, double* __restrict__ y,
                                                            double* __restrict__ dot_out,
                                                            double* __restrict__ partials,
                                                            unsigned int* __restrict__ counters, unsigned slot,
                                                            unsigned heal, const KeParam K) {
  const int nx1 = nx + 1, ny1 = ny + 1;
  const long long nn = (long long)nx1 * ny1 * (nz + 1);
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double dot = 0.0;
  if (r < nn) {
    const int x = (int)(r % nx1);
    const long long t = r / nx1;
    const int yy = (int)(t % ny1), z = (int)(t / ny1);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (int ez = z - 1; ez <= z; ++ez) {
      if (ez < 0 || ez >= nz) continue;
      for (int ey = yy - 1; ey <= yy; ++ey) {
        if (ey < 0 || ey >= ny) continue;
        for (int ex = x - 1; ex <= x; ++ex) {
          if (ex < 0 || ex >= nx) continue;
          const double Ee = E[((long long)ex * ny + ey) * nz + ez];
          const int ka = vf::corner_k(x - ex, yy - ey, z - ez);
          double t0 = 0.0, t1 = 0.0, t2 = 0.0;
#pragma unroll
          for (int kb = 0; kb < 8; ++kb) {
            const int bx = (kb == 1 || kb == 2 || kb == 5 || kb == 6);
            const int by = (kb == 2 || kb == 3 || kb == 6 || kb == 7);
            const int bz = (kb >= 4);
            const long long m = 3 * ((ex + bx) + (long long)nx1 * ((ey + by) + (long long)ny1 * (ez + bz)));
            const double u0 = u[m], u1 = u[m + 1], u2 = u[m + 2];
            const int r0 = (3 * ka) * 24 + 3 * kb;
            t0 += K.k[r0] * u0 + K.k[r0 + 1] * u1 + K.k[r0 + 2] * u2;
            t1 += K.k[r0 + 24] * u0 + K.k[r0 + 25] * u1 + K.k[r0 + 26] * u2;
            t2 += K.k[r0 + 48] * u0 + K.k[r0 + 49] * u1 + K.k[r0 + 50] * u2;
          }
          a0 += Ee * t0; a1 += Ee * t1; a2 += Ee * t2;
        }
      }
    }
    const uint8_t mk = mask[r];
    a0 = (mk & 1) ? a0 : 0.0;
    a1 = (mk & 2) ? a1 : 0.0;
    a2 = (mk & 4) ? a2 : 0.0;
    y[3 * r] = a0; y[3 * r + 1] = a1; y[3 * r + 2] = a2;
    dot = u[3 * r] * a0 + u[3 * r + 1] * a1 + u[3 * r + 2] * a2;
  }
  finish_dot(dot, dot_out, partials, counters, slot, heal);
}

// Planes per chunk of the marching form: the split whose waves of two blocks
// per SM take the fewest steps (a chunk of n planes marches n + 2).
March march_plan(int nx, int ny, int nz) {
  March m;
  m.ntx = (nx + kMX - 1) / (kMX - 1);
  m.nty = (ny + kMY - 1) / (kMY - 1);
  const long long tiles = (long long)m.ntx * m.nty, planes = nz + 1, room = 2 * 148;
  m.steps = -1;
  m.zchunk = (int)planes;
  // (the most chunks of each number of waves; past eight or so waves more
  // chunks only add their two extra steps)
  for (long long w = (tiles + room - 1) / room, w1 = w + 10; w < w1; ++w) {
    const long long n = std::min(planes, std::max(1LL, w * room / tiles)), zc = (planes + n - 1) / n;
    const long long waves = (tiles * ((planes + zc - 1) / zc) + room - 1) / room;
    if (m.steps < 0 || waves * (zc + 2) < m.steps) {
      m.steps = waves * (zc + 2);
      m.zchunk = (int)zc;
    }
    if (tiles * n > 8 * room) break;
  }
  m.units = tiles * ((planes + m.zchunk - 1) / m.zchunk);
  return m;
}

// The current device and the address of g_noalloc_scratch on it; the first time
// on a device, with both kernels loaded (so that a later capture loads nothing).
int scratch_for_device(int* device, unsigned char** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return VF_ERR_NO_DEVICE;
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      vf::g_last_error = std::string("cudaGetSymbolAddress(g_noalloc_scratch): ") + cudaGetErrorString(e);
      return VF_ERR_CUDA;
    }
    cudaFuncAttributes at;
    if ((e = cudaFuncGetAttributes(&at, k_apply_noalloc)) != cudaSuccess) {
      vf::g_last_error = std::string("vf_apply_noalloc: ") + cudaGetErrorString(e);
      return VF_ERR_CUDA;
    }
    vf::kernel_prepare(g_march_ready, k_apply_march, kMarchSmem, kThreads);
    g_scratch_addr[dev] = (unsigned char*)p;
  }
  *device = dev;
  *out = g_scratch_addr[dev];
  return VF_OK;
}

}  // namespace

extern "C" int vf_apply_noalloc(int32_t nx, int32_t ny, int32_t nz, double nu, const double* E,
                                const uint8_t* free_mask, const double* u, double* y, double* u_dot_y,
                                void* stream) {
  if (nx < 1 || ny < 1 || nz < 1 || !E || !free_mask || !u || !y || !u_dot_y) {
    vf::g_last_error = "vf_apply_noalloc: invalid argument";
    return VF_ERR_ARG;
  }
  if (!(nu > -1.0 && nu < 0.5)) {
    vf::g_last_error = "vf_apply_noalloc: Poisson ratio must lie in (-1, 0.5)";
    return VF_ERR_ARG;
  }
  const long long nn = (long long)(nx + 1) * (ny + 1) * (nz + 1);
  if (nn > kMaxNodes) {
    vf::g_last_error = "vf_apply_noalloc: grid has " + std::to_string(nn) + " nodes; the fixed scratch array "
                       "supports at most " + std::to_string(kMaxNodes) + " ((nx+1)(ny+1)(nz+1) <= 8388608)";
    return VF_ERR_ARG;
  }
  {
    // [u, u + 3nn), [y, y + 3nn) and the one double at u_dot_y must be disjoint
    const uintptr_t bu = (uintptr_t)u, by = (uintptr_t)y, bd = (uintptr_t)u_dot_y;
    const uintptr_t len = (uintptr_t)(3 * nn) * sizeof(double);
    auto overlap = [](uintptr_t a0, uintptr_t a1, uintptr_t b0, uintptr_t b1) { return a0 < b1 && b0 < a1; };
    if (overlap(bu, bu + len, by, by + len) || overlap(bd, bd + sizeof(double), bu, bu + len) ||
        overlap(bd, bd + sizeof(double), by, by + len)) {
      vf::g_last_error = "vf_apply_noalloc: u, y and u_dot_y must not overlap";
      return VF_ERR_ARG;
    }
  }
  int dev = 0;
  unsigned char* base = nullptr;
  int rc = scratch_for_device(&dev, &base);
  if (rc) return rc;
  double* partials = (double*)base;
  unsigned int* counters = (unsigned int*)(base + sizeof(double) * kMaxBlocks);
  cudaStream_t st = (cudaStream_t)stream;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(st, &cap);
  unsigned slot = kRing, heal = kRing;
  if (e == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
    slot = g_call[dev].fetch_add(1) % kRing;
    heal = (slot + kRing / 2) % kRing;
  } else if (e == cudaSuccess) {
    e = cudaMemsetAsync(counters + slot, 0, sizeof(unsigned int), st);
  }
  if (e != cudaSuccess) {
    vf::g_last_error = std::string("vf_apply_noalloc: ") + cudaGetErrorString(e);
    return VF_ERR_CUDA;
  }
  // The marching form takes a step's time however many of its tiles' 31 x 7
  // columns are nodes of the grid, the gather form a node's and an element's
  // time: in us about 5 + 1.3 steps (waves of units, two more planes each than
  // they own) against 9 + 0.03 per 1,000 nodes + 0.07 per 1,000 elements, and
  // about 13 more on the host, half of which count.  Marching / gather form, the
  // kernels: 100x100x100 47 / 112, 10000x10x10 49 / 109, 30x6x1000 16 / 30, 15x7x4000 47 / 56,
  // 200x1x200 16.1 / 16.5; on the other side 7x7x8000 80 / 56, 1x200x200 36 / 19, 3x40x3000
  // 88 / 53, 1x1x100000 390 / 45, 2000000x1x1 1,081 / 315.
  const March m = march_plan(nx, ny, nz);
  const double gather_us = 9.0 + 3e-5 * (double)nn + 7e-5 * (double)nx * ny * nz + 8.0;
  if (m.units <= kMaxBlocks && 5.0 + 1.3 * (double)m.steps < gather_us) {
    vf::launch_k(k_apply_march, dim3((unsigned)m.units), dim3(kMX, kMY), kMarchSmem, st, nx, ny, nz, E,
                 free_mask, u, y, u_dot_y, partials, counters, slot, heal, vf::modal_constants(nu, false), m);
  } else {
    KeParam K;
    double tab[1728], b0[144];
    vf::hex8_tables(nu, tab, b0);
    for (int i = 0; i < 576; ++i) K.k[i] = tab[i];
    const int blocks = (int)((nn + kThreads - 1) / kThreads);
    vf::launch_k(k_apply_noalloc, blocks, kThreads, 0, st, nx, ny, nz, E, free_mask, u, y, u_dot_y, partials, counters,
                 slot, heal, K);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    vf::g_last_error = std::string("vf_apply_noalloc launch: ") + cudaGetErrorString(e);
    return VF_ERR_CUDA;
  }
  return VF_OK;
}
