// Device pieces shared by the kernels that apply assembled Galerkin levels
// (vf_stencil.cu, vf_wide.cu): 16-byte chunks of the symmetric
// scaled storages and the rows of a reach-R operator.
#pragma once

#include <cuda_fp16.h>
#include <string.h>

#include "vf_common.cuh"

namespace vf {

__device__ __forceinline__ bool inside(const Grid& g, int x, int y, int z) {
  return x >= 0 && x <= g.lx && y >= 0 && y <= g.ly && z >= 0 && z <= g.lz;
}

// position of value k < 6 of SymLayout in the diagonal block
__host__ __device__ constexpr int diag_r(int k) { return k < 3 ? 0 : (k < 5 ? 1 : 2); }
__host__ __device__ constexpr int diag_c(int k) { return k < 3 ? k : (k < 5 ? k - 2 : 2); }

// One 16-byte chunk of stencil values, unpacked to the accumulation type.
template <typename S, typename A> struct Chunk;
template <> struct Chunk<__half, float> {
  float v[8];
  __device__ __forceinline__ void load(const __half* base) {
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(base));
    const unsigned ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __half2 h;
      memcpy(&h, &ws[i], 4);
      const float2 f = __half22float2(h);
      v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
  }
};
template <> struct Chunk<float, float> {
  float v[4];
  __device__ __forceinline__ void load(const float* base) {
    const float4 w = __ldg(reinterpret_cast<const float4*>(base));
    v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
  }
};

// ---- rows of a reach-R operator (WideLayout) --------------------------------
// The linear storage offset of upper block u (positive), or 0 for the diagonal
// block and the padding slots past it.
template <typename L>
__device__ __forceinline__ int wide_shift(const Grid& g, int u) {
  constexpr int R = (L::W - 1) / 2, W = L::W, SC = L::NB / 2;
  if (u >= L::NU) return 0;
  const int s = SC + 1 + u;
  return ((s / (W * W) - R) * g.py + (s / W) % W - R) * g.px + s % W - R;
}

__device__ __forceinline__ uint4 ldg_chunk(const void* p) {
  // volatile: a batch's loads stay together, ahead of its arithmetic
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
template <typename S, typename A> __device__ __forceinline__ A chunk_value(const uint4& c, int i);
template <> __device__ __forceinline__ float chunk_value<__half, float>(const uint4& c, int i) {
  const unsigned w = i < 2 ? c.x : (i < 4 ? c.y : (i < 6 ? c.z : c.w));
  __half2 h;
  memcpy(&h, &w, 4);
  return (i & 1) ? __high2float(h) : __low2float(h);
}
template <> __device__ __forceinline__ float chunk_value<float, float>(const uint4& c, int i) {
  return __uint_as_float(i == 0 ? c.x : (i == 1 ? c.y : (i == 2 ? c.z : c.w)));
}
template <> __device__ __forceinline__ double chunk_value<double, double>(const uint4& c, int i) {
  return i == 0 ? __hiloint2double((int)c.y, (int)c.x) : __hiloint2double((int)c.w, (int)c.z);
}

// A batch of JB block slots J0 .. J0 + JB - 1 of lane `lane` (of L::G lanes) of
// node p: own block u = lane + G*J applied to node p + shift, and the transposed
// block u of node p - shift (lane and slot are the same there).  V(slot, vu, vd)
// gives D^1/2 u of those nodes; ghost nodes hold zeros, so no neighbour needs a
// test, only the address of the transposed block is kept in the array.  load()
// depends on nothing but the node, so it may stand ahead of the staging of u.
// In FP32 apply() adds a block's three products of a row as one sum, a row of the
// own block, then a column of the transposed one: the order is part of the result
// (summed product by product into acc, the FP32 V-cycle differed by 1e-7 and a
// two-material displacement to a residual of 1e-11 by up to 2e-9 inside the void).
// FP64 sums product by product, 2-3 % of its V-cycle faster (256x128x128 1,784 /
// 1,832 us), as its order moves results by rounding only.
template <typename S> struct WideBatch { static constexpr int JB = sizeof(S) == 2 ? 4 : 2; };
template <typename S, typename L, int JB> struct RowBatch {
  static constexpr int VPC = L::VPC;
  static constexpr int NC = (9 * JB + VPC - 2) / VPC + 1;    // own chunks JB blocks may straddle
  static constexpr int ND = (9 + VPC - 2) / VPC + 1;         // chunks a block may straddle
  uint4 co[NC], cd[JB][ND];

  template <int J0> __device__ __forceinline__ void load(const Grid& g, const S* __restrict__ stc, int p, int lane) {
    constexpr int C0 = 9 * J0 / VPC, C1 = (9 * (J0 + JB) - 1) / VPC;
    static_assert(C1 - C0 < NC, "chunks of a batch");
    const S* own = stc + L::off((long long)p * L::G + lane, 0);
#pragma unroll
    for (int c = C0; c <= C1; ++c) co[c - C0] = ldg_chunk(own + c * 32 * VPC);
#pragma unroll
    for (int j = 0; j < JB; ++j) {
      const int k0 = 9 * (J0 + j), q = p - wide_shift<L>(g, lane + L::G * (J0 + j));
      const S* base = stc + L::off((long long)(q < 0 ? 0 : q) * L::G + lane, 0);
#pragma unroll
      for (int c = 0; c < ND; ++c)
        if (k0 / VPC + c <= (k0 + 8) / VPC) cd[j][c] = ldg_chunk(base + (k0 / VPC + c) * 32 * VPC);
    }
  }
  template <int J0, typename A, typename VF> __device__ __forceinline__ void apply(int lane, A (&acc)[3], VF V) const {
    constexpr int C0 = 9 * J0 / VPC;
#pragma unroll
    for (int j = 0; j < JB; ++j) {
      const int k0 = 9 * (J0 + j);
      A vu[3], vd[3];
      V(J0 + j, vu, vd);
      if (lane + L::G * (J0 + j) >= L::NU) vd[0] = vd[1] = vd[2] = (A)0;   // the diagonal block is applied once
      A bu[9], bd[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        bu[k] = chunk_value<S, A>(co[(k0 + k) / VPC - C0], (k0 + k) % VPC);
        bd[k] = chunk_value<S, A>(cd[j][(k0 + k) / VPC - k0 / VPC], (k0 + k) % VPC);
      }
      if constexpr (sizeof(A) == 4) {
#pragma unroll
        for (int r = 0; r < 3; ++r) acc[r] += bu[3 * r] * vu[0] + bu[3 * r + 1] * vu[1] + bu[3 * r + 2] * vu[2];
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += bd[c] * vd[0] + bd[3 + c] * vd[1] + bd[6 + c] * vd[2];
      } else {
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            acc[r] += bu[3 * r + c] * vu[c];
            acc[c] += bd[3 * r + c] * vd[r];
          }
      }
    }
  }
};

}  // namespace vf
