// 3x3x3 convolutions of the learned preconditioner stage: BF16 operands,
// FP32 accumulation on the tensor cores, implicit GEMM.
//
// Activations are channels-last BF16 tensors [Z][Y][X][C] (C = 16, 32 or 64),
// zero outside the box (the halo loads fill zeros: "same" padding).  Weights
// are [27][COUT][CIN] BF16 (tap = (dz+1)*9 + (dy+1)*3 + (dx+1)), so the
// input-channel axis -- the GEMM K axis -- is contiguous.
//
// Forward and backward-data (the forward of dY with the weights transposed
// and the taps mirrored) run on tcgen05 with TMEM accumulators
// (vf_nn_tc.cu); this file keeps the dispatch and the weight gradient.
//
// Backward-weight: dW[tap][co][ci] = sum_v dY[v][co] X[v + off(tap)][ci] is a
// GEMM with M = co, N = ci and K = voxels (mma.m16n8k16).  A CTA takes a group
// of taps and a strided set of voxel tiles; both operands come out of shared
// memory through ldmatrix.trans.  A warp keeps 16 co x 16 ci for every tap of
// the group in registers, so a row of 16 voxels costs one load of dY and one of
// X per tap for two products per tap (one tap, 8 ci at a time and both operands
// loaded for each product, the shared-memory pipe was the bound: 32-32
// channels on 68x52x36 voxels 127 us); with few channels the warps share the
// rows of a tile.  Per-CTA partial sums are reduced in a fixed order
// (deterministic).
#include <cuda_bf16.h>

#include <atomic>

#include "vf_common.cuh"
#include "vf_nn.cuh"

namespace vf {

namespace {

using bf16 = __nv_bfloat16;

constexpr int OTX = 16, OTY = 8, OTZ = 2;                 // output tile
constexpr int HTX = OTX + 2, HTY = OTY + 2, HTZ = OTZ + 2;
constexpr int NHALO = HTX * HTY * HTZ;                     // 720
constexpr int NTHREADS = 256;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm_x4_t(unsigned a, unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(a));
}
__device__ __forceinline__ void mma16816(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                         unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Load the (16 x 8 x 2 + halo) input box of a tile into shared memory,
// zero outside [0,X) x [0,Y) x [0,Z).  16-byte chunks.
template <int C, int CP>
__device__ __forceinline__ void load_halo(bf16* s, const bf16* __restrict__ g, int X, int Y, int Z, int X0, int Y0,
                                          int Z0) {
  constexpr int CH = C / 8;
  for (int i = threadIdx.x; i < NHALO * CH; i += NTHREADS) {
    const int v = i / CH, c = i - v * CH;
    const int hx = v % HTX, hy = (v / HTX) % HTY, hz = v / (HTX * HTY);
    const int x = X0 - 1 + hx, y = Y0 - 1 + hy, z = Z0 - 1 + hz;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (x >= 0 && x < X && y >= 0 && y < Y && z >= 0 && z < Z)
      val = __ldg(reinterpret_cast<const uint4*>(g + (((long long)z * Y + y) * X + x) * C) + c);
    *reinterpret_cast<uint4*>(s + v * CP + c * 8) = val;
  }
}

__device__ __forceinline__ int halo_index(int hx, int hy, int hz) { return (hz * HTY + hy) * HTX + hx; }

// ---------------------------------------------------------------------------
template <int CIN, int COUT>
struct WgradCfg {
  static constexpr int MT = COUT / 16, NP = CIN / 16, COMB = MT * NP;   // 16 x 16 blocks of (co, ci)
  static constexpr int CPW = COMB <= 8 ? 1 : COMB / 8;                  // blocks per warp
  static constexpr int KS = COMB < 8 ? 8 / COMB : 1;                    // warps sharing a block: rows of the tile
  static constexpr int TAPS = CPW == 1 ? 9 : 3;                         // 8 CPW TAPS accumulators per thread
  static constexpr int DP = COUT + 8;                                   // smem stride of a dY voxel
  static constexpr size_t smem() {
    return sizeof(bf16) * ((size_t)NHALO * (CIN + 8) + (size_t)OTX * OTY * OTZ * DP);
  }
  static_assert(KS == 1 || sizeof(float) * TAPS * COUT * CIN <= smem(), "the shared sum reuses the tile's memory");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(NTHREADS, 2)
    k_conv3_wgrad(const bf16* __restrict__ x, const bf16* __restrict__ dy, float* __restrict__ partial, int X, int Y,
                  int Z) {
  using Cfg = WgradCfg<CIN, COUT>;
  constexpr int CP = CIN + 8, DP = Cfg::DP, TAPS = Cfg::TAPS, KS = Cfg::KS, CPW = Cfg::CPW;
  extern __shared__ __align__(16) unsigned char smem[];
  bf16* sX = reinterpret_cast<bf16*>(smem);
  bf16* sD = sX + NHALO * CP;   // [256 tile voxels][DP], voxel = (tz*8 + ty)*16 + tx
  const int tx = (X + OTX - 1) / OTX, ty = (Y + OTY - 1) / OTY, tz = (Z + OTZ - 1) / OTZ;
  const int ntiles = tx * ty * tz;
  const int tap0 = blockIdx.y * TAPS;
  const int ddz = tap0 / 9, ddy0 = tap0 / 3 % 3;   // halo offsets (d + 1) of the group's first tap
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int comb0 = KS > 1 ? warp % Cfg::COMB : warp, part = KS > 1 ? warp / Cfg::COMB : 0;
  float acc[CPW][TAPS][2][4];
#pragma unroll
  for (int q = 0; q < CPW; ++q)
#pragma unroll
    for (int t = 0; t < TAPS; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[q][t][h][k] = 0.f;
  // A = dY^T (m = co, k = voxel), from [voxel][co]: ldmatrix.trans, row = voxel
  const int a_v = (lane & 7) + ((lane >> 4) & 1) * 8;
  const int a_c = ((lane >> 3) & 1) * 8;
  // B = X shifted (k = voxel, n = ci), from [voxel][ci]: two 8-channel halves per load
  const int b_v = (lane & 7) + ((lane >> 3) & 1) * 8;
  const int b_c = (lane >> 4) * 8;

#pragma unroll 1
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int X0 = (t % tx) * OTX, Y0 = ((t / tx) % ty) * OTY, Z0 = (t / (tx * ty)) * OTZ;
    __syncthreads();
    load_halo<CIN, CP>(sX, x, X, Y, Z, X0, Y0, Z0);
    {
      constexpr int CH = COUT / 8;
      for (int i = threadIdx.x; i < OTX * OTY * OTZ * CH; i += NTHREADS) {
        const int v = i / CH, c = i - v * CH;
        const int vx = v % OTX, vy = (v / OTX) % OTY, vz = v / (OTX * OTY);
        const int gx = X0 + vx, gy = Y0 + vy, gz = Z0 + vz;
        uint4 val = make_uint4(0u, 0u, 0u, 0u);
        if (gx < X && gy < Y && gz < Z)
          val = __ldg(reinterpret_cast<const uint4*>(dy + (((long long)gz * Y + gy) * X + gx) * COUT) + c);
        *reinterpret_cast<uint4*>(sD + v * DP + c * 8) = val;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int row = part; row < OTY * OTZ; row += KS) {
      const int ry = row % OTY, rz = row / OTY;
#pragma unroll
      for (int q = 0; q < CPW; ++q) {
        const int comb = comb0 + 8 * q, mt = comb / Cfg::NP, np = comb % Cfg::NP;
        unsigned a0, a1, a2, a3;
        ldsm_x4_t(smem_u32(sD + (row * OTX + a_v) * DP + mt * 16 + a_c), a0, a1, a2, a3);
        const unsigned xb = smem_u32(sX + halo_index(b_v, ry + ddy0, rz + ddz) * CP + np * 16 + b_c);
#pragma unroll
        for (int tap = 0; tap < TAPS; ++tap) {
          unsigned b0, b1, b2, b3;
          ldsm_x4_t(xb + (unsigned)(halo_index(tap % 3, tap / 3, 0) * CP * sizeof(bf16)), b0, b1, b2, b3);
          mma16816(acc[q][tap][0], a0, a1, a2, a3, b0, b1);
          mma16816(acc[q][tap][1], a0, a1, a2, a3, b2, b3);
        }
      }
    }
  }
  // partial[block][tap][co][ci] for the taps of this group
  const int g = lane >> 2, tig = lane & 3;
  float* dst = partial + (long long)blockIdx.x * 27 * COUT * CIN + (long long)tap0 * COUT * CIN;
  float* sum = reinterpret_cast<float*>(smem);
#pragma unroll 1
  for (int k = 0; k < KS; ++k) {
    if (KS > 1) __syncthreads();
    if (KS > 1 && part != k) continue;
#pragma unroll
    for (int q = 0; q < CPW; ++q) {
      const int comb = comb0 + 8 * q, mt = comb / Cfg::NP, np = comb % Cfg::NP;
#pragma unroll
      for (int tap = 0; tap < TAPS; ++tap)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int co = mt * 16 + g, ci = np * 16 + h * 8 + 2 * tig;
          float* d = (KS > 1 ? sum : dst) + ((long long)tap * COUT + co) * CIN + ci;
          const float* v = acc[q][tap][h];
          const bool add = KS > 1 && k > 0;
          d[0] = add ? d[0] + v[0] : v[0];
          d[1] = add ? d[1] + v[1] : v[1];
          d[8 * CIN] = add ? d[8 * CIN] + v[2] : v[2];
          d[8 * CIN + 1] = add ? d[8 * CIN + 1] + v[3] : v[3];
        }
    }
  }
  if (KS > 1) {
    __syncthreads();
    for (int i = threadIdx.x; i < TAPS * COUT * CIN; i += NTHREADS) dst[i] = sum[i];
  }
}

// Sums of the per-CTA partials in a fixed order, in FP64: 8 threads per value
// take every eighth partial (one thread per value walked all of them, 21 us for
// 27,648 values of 148 partials).
__global__ void __launch_bounds__(256) k_reduce_partials(const float* __restrict__ partial, int nparts, long long n,
                                                         float* __restrict__ out, int accumulate) {
  __shared__ double s[8][33];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const long long i = blockIdx.x * 32LL + lane;
  double v = 0.0;
  if (i < n) {
#pragma unroll 4
    for (int b = grp; b < nparts; b += 8) v += __ldg(partial + (long long)b * n + i);
  }
  s[grp][lane] = v;
  __syncthreads();
  if (grp == 0 && i < n) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += s[k][lane];
    out[i] = accumulate ? out[i] + (float)t : (float)t;
  }
}

// Bias gradient: column sums of dY.  A thread keeps 8 consecutive channels (16
// bytes a voxel) of every gridDim-th group of voxels; a block's threads of the
// same channels, then the blocks, are summed in a fixed order and in FP64, so
// only the thread's own few additions and a block's one rounding are FP32 (all in
// FP32: 1.2e-7 from FP64 on 68x52x36 voxels, a pairwise FP32 sum 0.9e-7, now 0.3e-7).  (As a
// conversion to FP32 and a generic reduction: 35 us for 32 channels on
// 68x52x36 voxels, the bytes take 1.5.)
constexpr int kBiasBlocks = 148;
template <int COUT>
__global__ void __launch_bounds__(NTHREADS) k_bias_grad(const bf16* __restrict__ dy, long long nvox,
                                                        float* __restrict__ partial) {
  constexpr int CH = COUT / 8, VOX = NTHREADS / CH;
  __shared__ float s[NTHREADS][9];
  const int ch = threadIdx.x % CH, v0 = threadIdx.x / CH;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (long long v = (long long)blockIdx.x * VOX + v0; v < nvox; v += (long long)gridDim.x * VOX) {
    const uint4 p = __ldg(reinterpret_cast<const uint4*>(dy + v * COUT) + ch);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&p);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = __bfloat1622float2(h[k]);
      acc[2 * k] += f.x;
      acc[2 * k + 1] += f.y;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s[threadIdx.x][k] = acc[k];
  __syncthreads();
  if (threadIdx.x < COUT) {
    const int c = threadIdx.x;
    double t = 0.0;
    for (int v = 0; v < VOX; ++v) t += s[v * CH + c / 8][c % 8];
    partial[(long long)blockIdx.x * COUT + c] = (float)t;
  }
}

// Partials (CTAs of a tap group) of a weight gradient whose `ks` warps share a
// block of channels: whole waves of resident CTAs, and at least so many that a
// warp adds up no more rows than with 148 partials of one warp each.  The FP32
// accumulators of the MMA truncate, so the error grows with the rows added up.
// 36 x 52 x 68 voxels, one wave / by this rule, error against FP64 and time: 64-64
// channels 32 partials 7.0e-6, 259 us / 164 partials 5.3e-7, 297 us; 64-32 98
// partials 1.8e-6, 110 us / 197 partials 5.1e-7, 119 us.
int wgrad_parts(int ks, int groups, int per_sm) {
  const int need = (148 + ks - 1) / ks, room = 148 * std::min(per_sm, 2);
  return room * ((need * groups + room - 1) / room) / groups;
}

template <int CIN, int COUT>
int conv_wgrad_t(const void* x, const void* dy, float* dw, float* work, size_t work_bytes, int X, int Y, int Z,
                 int accumulate, cudaStream_t st) {
  using Cfg = WgradCfg<CIN, COUT>;
  const size_t per = sizeof(float) * 27 * COUT * CIN;
  const long long tiles = (long long)((X + OTX - 1) / OTX) * ((Y + OTY - 1) / OTY) * ((Z + OTZ - 1) / OTZ);
  constexpr size_t smem = Cfg::smem();
  static std::atomic<int> per_dev[kMaxDevices];
  const int per_sm = kernel_prepare(per_dev, k_conv3_wgrad<CIN, COUT>, smem, NTHREADS);
  constexpr int groups = 27 / Cfg::TAPS;
  long long nb = std::min<long long>(tiles, wgrad_parts(Cfg::KS, groups, per_sm));
  nb = std::min<long long>(nb, (long long)(work_bytes / per));
  if (nb < 1) return -1;
  launch_k(k_conv3_wgrad<CIN, COUT>, dim3((unsigned)nb, groups), dim3(NTHREADS), smem, st,
           (const bf16*)x, (const bf16*)dy, work, X, Y, Z);
  const long long n = 27LL * COUT * CIN;
  launch_k(k_reduce_partials, dim3((unsigned)((n + 31) / 32)), dim3(256), 0, st, (const float*)work, (int)nb, n,
           dw, accumulate);
  return 0;
}

}  // namespace

#define VF_NN_PAIRS(F) F(16, 16) F(16, 32) F(32, 16) F(32, 32) F(32, 64) F(64, 32) F(64, 64)

size_t nn_wgrad_work_bytes(int cin, int cout, int X, int Y, int Z) {
  const long long tiles = (long long)((X + OTX - 1) / OTX) * ((Y + OTY - 1) / OTY) * ((Z + OTZ - 1) / OTZ);
  long long parts = 148;
#define VF_NN_PARTS(I, O)                                                                   \
  if (cin == I && cout == O) {                                                              \
    using C = WgradCfg<I, O>;                                                               \
    parts = std::max(wgrad_parts(C::KS, 27 / C::TAPS, 1), wgrad_parts(C::KS, 27 / C::TAPS, 2)); \
  }
  VF_NN_PAIRS(VF_NN_PARTS)
#undef VF_NN_PARTS
  return sizeof(float) * 27 * (size_t)cin * cout * (size_t)std::max<long long>(1, std::min<long long>(tiles, parts));
}

template <int CIN, int COUT> int conv_forward_tc(const NnConvArgs& a, cudaStream_t st);   // vf_nn_tc.cu

int nn_conv_forward(int cin, int cout, const NnConvArgs& a, cudaStream_t st) {
#define VF_NN_FWD(I, O) \
  if (cin == I && cout == O) return conv_forward_tc<I, O>(a, st);
  VF_NN_PAIRS(VF_NN_FWD)
#undef VF_NN_FWD
  return -1;
}

int nn_conv_wgrad(int cin, int cout, const void* x, const void* dy, float* dw, float* work, size_t work_bytes, int X,
                  int Y, int Z, int accumulate, cudaStream_t st) {
#define VF_NN_WG(I, O) \
  if (cin == I && cout == O) return conv_wgrad_t<I, O>(x, dy, dw, work, work_bytes, X, Y, Z, accumulate, st);
  VF_NN_PAIRS(VF_NN_WG)
#undef VF_NN_WG
  return -1;
}

}  // namespace vf

// ---------------------------------------------------------------------------
// C-ABI
// ---------------------------------------------------------------------------
#include "../../include/voxfea.h"

namespace {
// The kernels move activations, weights and results 16 bytes at a time.
bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr, const void* d = nullptr) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15) == 0;
}
}  // namespace

extern "C" {

int vf_nn_conv3d_forward(const void* in, const void* w, const float* bias, const void* skip, int32_t relu, void* out,
                         float* out_f32, int32_t X, int32_t Y, int32_t Z, int32_t cin, int32_t cout, void* stream) {
  if (!in || !w || (!out && !out_f32) || X < 1 || Y < 1 || Z < 1 || !aligned16(in, w, out_f32 ? out_f32 : out))
    return VF_ERR_ARG;
  vf::NnConvArgs a{in, w, bias, skip, nullptr, out, out_f32, X, Y, Z, relu ? 1 : 0};
  if (vf::nn_conv_forward(cin, cout, a, (cudaStream_t)stream)) return VF_ERR_ARG;
  return cudaPeekAtLastError() == cudaSuccess ? VF_OK : VF_ERR_CUDA;
}

int vf_nn_conv3d_backward_data(const void* dy, const void* w_t, const void* gate, void* dx, int32_t X, int32_t Y,
                               int32_t Z, int32_t cin, int32_t cout, void* stream) {
  if (!dy || !w_t || !dx || X < 1 || Y < 1 || Z < 1 || !aligned16(dy, w_t, dx)) return VF_ERR_ARG;
  vf::NnConvArgs a{dy, w_t, nullptr, nullptr, gate, dx, nullptr, X, Y, Z, 0};
  if (vf::nn_conv_forward(cout, cin, a, (cudaStream_t)stream)) return VF_ERR_ARG;
  return cudaPeekAtLastError() == cudaSuccess ? VF_OK : VF_ERR_CUDA;
}

int vf_nn_conv3d_backward_weight(const void* x, const void* dy, float* dw, int32_t accumulate, float* work,
                                 size_t work_bytes, int32_t X, int32_t Y, int32_t Z, int32_t cin, int32_t cout,
                                 void* stream) {
  if (!x || !dy || !dw || !work || X < 1 || Y < 1 || Z < 1 || !aligned16(x, dy)) return VF_ERR_ARG;
  if (vf::nn_conv_wgrad(cin, cout, x, dy, dw, work, work_bytes, X, Y, Z, accumulate, (cudaStream_t)stream))
    return VF_ERR_ARG;
  return cudaPeekAtLastError() == cudaSuccess ? VF_OK : VF_ERR_CUDA;
}

int vf_nn_conv3d_backward_bias(const void* dy, float* db, float* work, size_t work_bytes, int64_t nvox, int32_t cout,
                               void* stream) {
  using namespace vf;
  if (!dy || !db || !work || nvox < 1 || work_bytes < sizeof(float) * kBiasBlocks * (size_t)cout || !aligned16(dy))
    return VF_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const bf16* d = (const bf16*)dy;
  const int nb = (int)std::min<long long>(kBiasBlocks, (nvox * cout / 8 + NTHREADS - 1) / NTHREADS);
  if (cout == 16) launch_k(k_bias_grad<16>, nb, NTHREADS, 0, st, d, (long long)nvox, work);
  else if (cout == 32) launch_k(k_bias_grad<32>, nb, NTHREADS, 0, st, d, (long long)nvox, work);
  else if (cout == 64) launch_k(k_bias_grad<64>, nb, NTHREADS, 0, st, d, (long long)nvox, work);
  else return VF_ERR_ARG;
  launch_k(k_reduce_partials, (cout + 31) / 32, 256, 0, st, (const float*)work, nb, (long long)cout, db, 0);
  return cudaPeekAtLastError() == cudaSuccess ? VF_OK : VF_ERR_CUDA;
}

size_t vf_nn_wgrad_workspace(int32_t cin, int32_t cout, int32_t X, int32_t Y, int32_t Z) {
  return vf::nn_wgrad_work_bytes(cin, cout, X, Y, Z);
}

}  // extern "C"
