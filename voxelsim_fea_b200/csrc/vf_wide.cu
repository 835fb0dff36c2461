// Wide Galerkin levels: the coarse space with a smoothed prolongation.
//
// The robust hierarchy's coarse operators A_{l+1} = D P^T A_l P D use the
// reference's trilinear P (core/multigrid.py:42-73).  On the transfer from a
// Galerkin level l to l+1 this library can instead use the smoothed
// prolongation of smoothed aggregation,
//
//     P_s = D_l (I - c_l D_l^-1 A_l) P,     c_l = (4/3) / lambda_l,
//
// lambda_l the padded power-iteration estimate of lambda_max(D_l^-1 A_l),
// and A_{l+1} = D_{l+1} P_s^T A_l P_s D_{l+1}.  The smoothed basis functions
// reach one fine node further, so the coarse operator couples each node with
// the nodes up to two (in general: R) coarse spacings away: 125 blocks of
// 3x3 per node instead of 27.  The transfers themselves need no new kernel
// (vf_solver.cu): restriction P_s^T r = P^T (r - c A (Minv r)) and
// prolongation x += P_s e = t - c Minv A t (t = P e) are the level's own
// residual and sweep kernels.
//
// Set-up (FP64, once per set_material), for the transfer l -> l+1:
//   k_prolong_blocks  the 3x3 blocks P_s[i][J] of every fine node i
//                     ((Pr+1)^3 coarse slots per node, stored entry-major
//                     and slot-fastest per node; Pr = 1 + R_l when
//                     smoothed, 1 for the trilinear P);
//   k_rap_b           B = A_l P_s, (Pr+R_l+1)^3 coarse slots per fine node;
//   k_rap_c           the diagonal and upper blocks of A_{l+1} = P_s^T B, one
//                     CTA per coarse node, P_s[.][I] staged in shared memory;
//   k_wide_mirror     the lower blocks as the neighbours' transposed upper
//                     ones (the coarse operator is exactly symmetric);
//   k_wide_mask_diag  D_{l+1} = DOFs with a positive diagonal, rows / columns
//                     of the others zeroed, inverse diagonal.
// Full stencils: st[(s*9 + 3r + c) * n + p], s = ((dz+R)*W + (dy+R))*W + (dx+R),
// W = 2R+1: coupling of DOF r of node p with DOF c of node p + (dx,dy,dz).
//
// Apply (V-cycle), also of the 27-block levels in FP64 and of the small ones:
// symmetric, diagonally scaled storage -- the diagonal block and the upper
// blocks s > center (9 values each) of A~ = D^-1/2 A D^-1/2, FP16 for the
// FP32 V-cycle, warp-chunked so a warp loads one 16-byte chunk of 32
// consecutive nodes at once; the lower blocks are read transposed from the
// neighbour that stores them.
#include <cuda_fp16.h>

#include <type_traits>

#include "vf_common.cuh"
#include "vf_levelops.cuh"
#include "vf_reduce.cuh"

namespace vf {

namespace {

__host__ __device__ constexpr int wide_w(int R) { return 2 * R + 1; }
__host__ __device__ constexpr int wide_nb(int R) { return (2 * R + 1) * (2 * R + 1) * (2 * R + 1); }

// 1-D trilinear weight of a coarse node at fine offset d
__device__ __forceinline__ double tw(int d) { return d == 0 ? 1.0 : ((d == 1 || d == -1) ? 0.5 : 0.0); }
// ceil(v / 2) for any sign
__device__ __forceinline__ int ceil_half(int v) { return v >= 0 ? (v + 1) / 2 : -((-v) / 2); }

__device__ __forceinline__ void interior_xyz(const Grid& g, long long t, int& x, int& y, int& z) {
  const int nx1 = g.lx + 1, ny1 = g.ly + 1;
  x = (int)(t % nx1);
  const long long r = t / nx1;
  y = (int)(r % ny1);
  z = (int)(r / ny1);
}

__device__ __forceinline__ void decode(const Grid& g, int p, int& x, int& y, int& z) {
  x = p % g.px - 1;
  const int t = p / g.px;
  y = t % g.py - 1;
  z = t / g.py - 1;
}

inline int blocks_for(long long n, int threads, long long cap = 148LL * 64) {
  long long b = (n + threads - 1) / threads;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

// ---- set-up ----------------------------------------------------------------

// CTAs of the set-up products handle NG consecutive interior nodes x NS
// slots (NG = kSetupThreads / NS); the level-l blocks of those nodes are
// staged once in shared memory instead of being re-read by every slot.
constexpr int kSetupThreads = 256;

// Stage the full stencil blocks of nodes [n0, n0 + NG) in sA[(node * NB + s) * 9 + k].
__device__ __forceinline__ void stage_blocks(const Grid& f, const double* __restrict__ stf, int NB, long long n0,
                                             int NG, long long nint, double* sA) {
  const long long nf = f.n;
  for (int e = threadIdx.x; e < NG * NB * 9; e += blockDim.x) {
    const int nl = e / (NB * 9), rem = e % (NB * 9), s = rem / 9, k = rem % 9;
    double v = 0.0;
    if (n0 + nl < nint) {
      int x, y, z;
      interior_xyz(f, n0 + nl, x, y, z);
      v = stf[((long long)s * 9 + k) * nf + f.idx(x, y, z)];
    }
    sA[e] = v;
  }
}

// P_s[i][J] per fine interior node i and coarse slot (ax, ay, az), J = jlo(i) + a,
// jlo = ceil((i - Pr) / 2) per axis; psb[(p * 9 + 3r + c) * NS + slot] (slot fastest:
// the consecutive slots a warp reads or writes are consecutive words).
// smoothed: *cdev != 0 (the blocks of A staged); else the trilinear D P.
__global__ void __launch_bounds__(kSetupThreads) k_prolong_blocks(Grid f, const double* __restrict__ stf, int Rf,
                                                                  const uint8_t* __restrict__ fm,
                                                                  const double* __restrict__ minvf,
                                                                  const double* __restrict__ cdev, int Pr, Grid c,
                                                                  double* __restrict__ psb) {
  extern __shared__ double sA[];
  const int NA = Pr + 1, NS = NA * NA * NA, NG = kSetupThreads / NS;
  const int W = wide_w(Rf), NB = wide_nb(Rf);
  const long long nint = (long long)(f.lx + 1) * (f.ly + 1) * (f.lz + 1);
  const double cc = cdev ? *cdev : 0.0;
  for (long long n0 = (long long)blockIdx.x * NG; n0 < nint; n0 += (long long)gridDim.x * NG) {
    if (cdev) {
      __syncthreads();
      stage_blocks(f, stf, NB, n0, NG, nint, sA);
      __syncthreads();
    }
    const int nl = threadIdx.x / NS, slot = threadIdx.x % NS;
    if (nl >= NG || n0 + nl >= nint) continue;
    int x, y, z;
    interior_xyz(f, n0 + nl, x, y, z);
    const int p = f.idx(x, y, z);
    const int ax = slot % NA, ay = (slot / NA) % NA, az = slot / (NA * NA);
    const int Jx = ceil_half(x - Pr) + ax, Jy = ceil_half(y - Pr) + ay, Jz = ceil_half(z - Pr) + az;
    double blk[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) blk[k] = 0.0;
    if (inside(c, Jx, Jy, Jz)) {
      const uint8_t m = fm[p];
      const double w = tw(x - 2 * Jx) * tw(y - 2 * Jy) * tw(z - 2 * Jz);
#pragma unroll
      for (int r = 0; r < 3; ++r)
        if ((m >> r) & 1) blk[4 * r] = w;
      if (cdev && cc != 0.0 && m) {
        // - c Minv_i sum_d A[i][d] w(i + d, J)
        double acc[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[k] = 0.0;
        const double* A = sA + (long long)nl * NB * 9;
        for (int s = 0; s < NB; ++s) {
          const int dx = s % W - Rf, dy = (s / W) % W - Rf, dz = s / (W * W) - Rf;
          const double wk = tw(x + dx - 2 * Jx) * tw(y + dy - 2 * Jy) * tw(z + dz - 2 * Jz);
          if (wk == 0.0 || !inside(f, x + dx, y + dy, z + dz)) continue;
#pragma unroll
          for (int k = 0; k < 9; ++k) acc[k] += wk * A[s * 9 + k];
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const double mr = minvf[3LL * p + r];
#pragma unroll
          for (int k = 0; k < 3; ++k) blk[3 * r + k] -= cc * mr * acc[3 * r + k];
        }
      }
    }
    double* out = psb + (long long)p * NS * 9 + slot;
#pragma unroll
    for (int k = 0; k < 9; ++k) out[k * NS] = blk[k];
  }
}

// B[k][J] = sum_d A[k][d] P_s[k + d][J] per fine interior node k and coarse
// slot b, J = ceil((k - Pr - Rf) / 2) + b per axis; bsb[(p * 9 + 3r + c) * NSB + b].
__global__ void __launch_bounds__(kSetupThreads) k_rap_b(Grid f, const double* __restrict__ stf, int Rf,
                                                         const double* __restrict__ psb, int Pr, Grid c,
                                                         double* __restrict__ bsb) {
  extern __shared__ double sA[];
  const int NA = Pr + 1, NS = NA * NA * NA;
  const int NBA = Pr + Rf + 1, NSB = NBA * NBA * NBA, NG = kSetupThreads / NSB;
  const int W = wide_w(Rf), NB = wide_nb(Rf);
  const long long nint = (long long)(f.lx + 1) * (f.ly + 1) * (f.lz + 1);
  for (long long n0 = (long long)blockIdx.x * NG; n0 < nint; n0 += (long long)gridDim.x * NG) {
    __syncthreads();
    stage_blocks(f, stf, NB, n0, NG, nint, sA);
    __syncthreads();
    const int nl = threadIdx.x / NSB, b = threadIdx.x % NSB;
    if (nl >= NG || n0 + nl >= nint) continue;
    int x, y, z;
    interior_xyz(f, n0 + nl, x, y, z);
    const int p = f.idx(x, y, z);
    const int Jx = ceil_half(x - Pr - Rf) + b % NBA, Jy = ceil_half(y - Pr - Rf) + (b / NBA) % NBA;
    const int Jz = ceil_half(z - Pr - Rf) + b / (NBA * NBA);
    double acc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k] = 0.0;
    if (inside(c, Jx, Jy, Jz)) {
      const double* As = sA + (long long)nl * NB * 9;
      for (int s = 0; s < NB; ++s) {
        const int ix = x + s % W - Rf, iy = y + (s / W) % W - Rf, iz = z + s / (W * W) - Rf;
        if (!inside(f, ix, iy, iz)) continue;
        const int ax = Jx - ceil_half(ix - Pr), ay = Jy - ceil_half(iy - Pr), az = Jz - ceil_half(iz - Pr);
        if (ax < 0 || ax > Pr || ay < 0 || ay > Pr || az < 0 || az > Pr) continue;
        const double* P = psb + (long long)f.idx(ix, iy, iz) * NS * 9 + (az * NA + ay) * NA + ax;
        const double* A = As + s * 9;
        double Pv[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) Pv[k] = P[k * NS];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int cc = 0; cc < 3; ++cc)
            acc[3 * r + cc] += A[3 * r] * Pv[cc] + A[3 * r + 1] * Pv[3 + cc] + A[3 * r + 2] * Pv[6 + cc];
      }
    }
    double* out = bsb + (long long)p * NSB * 9 + b;
#pragma unroll
    for (int k = 0; k < 9; ++k) out[k * NSB] = acc[k];
  }
}

// A_{l+1}[I][I + D] = sum_i P_s[i][I]^T B[i][I + D] for the diagonal and the
// upper offsets D of reach Rc: one CTA per coarse interior node I, P_s[.][I]
// of the (2Pr+1)^3 fine nodes around 2I in shared memory, one thread per D.
constexpr int kRapThreads = 64;
__global__ void __launch_bounds__(kRapThreads) k_rap_c(Grid f, int Rf, const double* __restrict__ psb, int Pr,
                                                       const double* __restrict__ bsb, Grid c, int Rc,
                                                       double* __restrict__ stc) {
  extern __shared__ double sps[];   // [(2Pr+1)^3][9]
  const int NA = Pr + 1, NS = NA * NA * NA;
  const int NBA = Pr + Rf + 1, NSB = NBA * NBA * NBA;
  const int WI = 2 * Pr + 1, NI = WI * WI * WI;
  const int Wc = wide_w(Rc), NBc = wide_nb(Rc), SC = NBc / 2;
  const long long nint = (long long)(c.lx + 1) * (c.ly + 1) * (c.lz + 1);
  const long long nc = c.n;
  for (long long node = blockIdx.x; node < nint; node += gridDim.x) {
    int X, Y, Z;
    interior_xyz(c, node, X, Y, Z);
    const int pI = c.idx(X, Y, Z);
    __syncthreads();   // the previous node's readers are done with sps
    for (int e = threadIdx.x; e < NI * 9; e += blockDim.x) {
      const int i = e / 9, k = e % 9;
      const int ix = 2 * X + i % WI - Pr, iy = 2 * Y + (i / WI) % WI - Pr, iz = 2 * Z + i / (WI * WI) - Pr;
      double v = 0.0;
      if (inside(f, ix, iy, iz)) {
        const int ax = X - ceil_half(ix - Pr), ay = Y - ceil_half(iy - Pr), az = Z - ceil_half(iz - Pr);
        v = psb[((long long)f.idx(ix, iy, iz) * 9 + k) * NS + (az * NA + ay) * NA + ax];
      }
      sps[e] = v;
    }
    __syncthreads();
    for (int u = threadIdx.x; u <= SC; u += blockDim.x) {
      const int s = SC + u;   // center and upper offsets
      const int Dx = s % Wc - Rc, Dy = (s / Wc) % Wc - Rc, Dz = s / (Wc * Wc) - Rc;
      const int Jx = X + Dx, Jy = Y + Dy, Jz = Z + Dz;
      double acc[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) acc[k] = 0.0;
      if (inside(c, Jx, Jy, Jz)) {
        for (int i = 0; i < NI; ++i) {
          const int ix = 2 * X + i % WI - Pr, iy = 2 * Y + (i / WI) % WI - Pr, iz = 2 * Z + i / (WI * WI) - Pr;
          if (!inside(f, ix, iy, iz)) continue;
          const int bx = Jx - ceil_half(ix - Pr - Rf), by = Jy - ceil_half(iy - Pr - Rf);
          const int bz = Jz - ceil_half(iz - Pr - Rf);
          if (bx < 0 || bx >= NBA || by < 0 || by >= NBA || bz < 0 || bz >= NBA) continue;
          const double* P = sps + i * 9;
          const double* B = bsb + (long long)f.idx(ix, iy, iz) * NSB * 9 + (bz * NBA + by) * NBA + bx;
          double Bv[9];
#pragma unroll
          for (int k = 0; k < 9; ++k) Bv[k] = B[k * NSB];
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int cc = 0; cc < 3; ++cc)
              acc[3 * r + cc] += P[r] * Bv[cc] + P[3 + r] * Bv[3 + cc] + P[6 + r] * Bv[6 + cc];
        }
      }
#pragma unroll
      for (int k = 0; k < 9; ++k) stc[((long long)s * 9 + k) * nc + pI] = acc[k];
    }
  }
}

// ---- set-up products with the reaches fixed at compile time ------------------
// The hierarchies this library builds use two (R_l, Pr) pairs: (1, 2) for the
// smoothed transfer from a 27-block level and (2, 1) for the trilinear
// transfer below a 125-block level, both giving R_{l+1} = 2.  The kernels
// below compute exactly the sums of k_prolong_blocks / k_rap_b (the same
// terms, added in the same order) but with W, NB and the slot counts as
// constants and the contributing offsets found per axis instead of by testing
// all NB of them: the generic kernels spend most of their time on runtime
// divisions and range tests, not on the FP64 products.  (The coarse product
// stays generic: a compile-time version held twice the registers and ran
// slower; so did a B product that staged the neighbours' P_s rows in shared
// memory.)

// Padded-storage index and interior coordinates of the interior nodes
// [n0, n0 + NG) of grid f (-1 past the end), for a CTA's staging.
template <int NG>
__device__ __forceinline__ void node_table(const Grid& f, long long n0, long long nint, int* sp) {
  if (threadIdx.x < NG) {
    int v = -1;
    if (n0 + threadIdx.x < nint) {
      int x, y, z;
      interior_xyz(f, n0 + threadIdx.x, x, y, z);
      v = f.idx(x, y, z);
    }
    sp[threadIdx.x] = v;
  }
}

template <int RF, int PR, bool SMOOTHED>
__global__ void __launch_bounds__(kSetupThreads) k_prolong_blocks_t(Grid f, const double* __restrict__ stf,
                                                                    const uint8_t* __restrict__ fm,
                                                                    const double* __restrict__ minvf,
                                                                    const double* __restrict__ cdev, Grid c,
                                                                    double* __restrict__ psb) {
  constexpr int NA = PR + 1, NS = NA * NA * NA, NG = kSetupThreads / NS;
  constexpr int W = 2 * RF + 1, NB = W * W * W;
  __shared__ double sA[SMOOTHED ? NG * NB * 9 : 1];
  __shared__ int sp[NG];
  const long long nint = (long long)(f.lx + 1) * (f.ly + 1) * (f.lz + 1);
  const long long nf = f.n;
  const double cc = SMOOTHED ? *cdev : 0.0;
  const int sxy = f.px * f.py;
  for (long long n0 = (long long)blockIdx.x * NG; n0 < nint; n0 += (long long)gridDim.x * NG) {
    __syncthreads();   // the previous group's readers are done with sA / sp
    node_table<NG>(f, n0, nint, sp);
    __syncthreads();
    if (SMOOTHED) {
      for (int e = threadIdx.x; e < NG * NB * 9; e += blockDim.x) {
        const int nl = e / (NB * 9), rem = e - nl * (NB * 9);
        const int p = sp[nl];
        sA[e] = p >= 0 ? stf[(long long)rem * nf + p] : 0.0;
      }
      __syncthreads();
    }
    const int nl = threadIdx.x / NS, slot = threadIdx.x - nl * NS;
    if (nl >= NG) continue;
    const int p = sp[nl];
    if (p < 0) continue;
    const int z = p / sxy - 1, rxy = p - (z + 1) * sxy, y = rxy / f.px - 1, x = rxy - (y + 1) * f.px - 1;
    const int ax = slot % NA, ay = (slot / NA) % NA, az = slot / (NA * NA);
    const int Jx = ceil_half(x - PR) + ax, Jy = ceil_half(y - PR) + ay, Jz = ceil_half(z - PR) + az;
    double blk[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) blk[k] = 0.0;
    if (inside(c, Jx, Jy, Jz)) {
      const uint8_t m = fm[p];
      const double w = tw(x - 2 * Jx) * tw(y - 2 * Jy) * tw(z - 2 * Jz);
#pragma unroll
      for (int r = 0; r < 3; ++r)
        if ((m >> r) & 1) blk[4 * r] = w;
      if (SMOOTHED && cc != 0.0 && m) {
        double wx[W], wy[W], wz[W];
#pragma unroll
        for (int d = 0; d < W; ++d) {
          const int ix = x + d - RF, iy = y + d - RF, iz = z + d - RF;
          wx[d] = (ix >= 0 && ix <= f.lx) ? tw(ix - 2 * Jx) : 0.0;
          wy[d] = (iy >= 0 && iy <= f.ly) ? tw(iy - 2 * Jy) : 0.0;
          wz[d] = (iz >= 0 && iz <= f.lz) ? tw(iz - 2 * Jz) : 0.0;
        }
        double acc[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[k] = 0.0;
        const double* A = sA + nl * NB * 9;
#pragma unroll
        for (int dz = 0; dz < W; ++dz) {
          if (wz[dz] == 0.0) continue;
#pragma unroll
          for (int dy = 0; dy < W; ++dy) {
            if (wy[dy] == 0.0) continue;
#pragma unroll
            for (int dx = 0; dx < W; ++dx) {
              if (wx[dx] == 0.0) continue;
              const double wk = wx[dx] * wy[dy] * wz[dz];
              const double* As = A + ((dz * W + dy) * W + dx) * 9;
#pragma unroll
              for (int k = 0; k < 9; ++k) acc[k] += wk * As[k];
            }
          }
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const double mr = minvf[3LL * p + r];
#pragma unroll
          for (int k = 0; k < 3; ++k) blk[3 * r + k] -= cc * mr * acc[3 * r + k];
        }
      }
    }
    double* out = psb + (long long)p * NS * 9 + slot;
#pragma unroll
    for (int k = 0; k < 9; ++k) out[k * NS] = blk[k];
  }
}

template <int RF, int PR>
__global__ void __launch_bounds__(kSetupThreads, 4) k_rap_b_t(Grid f, const double* __restrict__ stf,
                                                           const double* __restrict__ psb, Grid c,
                                                           double* __restrict__ bsb) {
  constexpr int NA = PR + 1, NS = NA * NA * NA;
  constexpr int NBA = PR + RF + 1, NSB = NBA * NBA * NBA, NG = kSetupThreads / NSB;
  constexpr int W = 2 * RF + 1, NB = W * W * W;
  __shared__ double sA[NG * NB * 9];
  __shared__ int sp[NG];
  const long long nint = (long long)(f.lx + 1) * (f.ly + 1) * (f.lz + 1);
  const long long nf = f.n;
  const int sxy = f.px * f.py;
  for (long long n0 = (long long)blockIdx.x * NG; n0 < nint; n0 += (long long)gridDim.x * NG) {
    __syncthreads();
    node_table<NG>(f, n0, nint, sp);
    __syncthreads();
    for (int e = threadIdx.x; e < NG * NB * 9; e += blockDim.x) {
      const int nl = e / (NB * 9), rem = e - nl * (NB * 9);
      const int p = sp[nl];
      sA[e] = p >= 0 ? stf[(long long)rem * nf + p] : 0.0;
    }
    __syncthreads();
    const int nl = threadIdx.x / NSB, b = threadIdx.x - nl * NSB;
    if (nl >= NG) continue;
    const int p = sp[nl];
    if (p < 0) continue;
    const int z = p / sxy - 1, rxy = p - (z + 1) * sxy, y = rxy / f.px - 1, x = rxy - (y + 1) * f.px - 1;
    const int Jx = ceil_half(x - PR - RF) + b % NBA, Jy = ceil_half(y - PR - RF) + (b / NBA) % NBA;
    const int Jz = ceil_half(z - PR - RF) + b / (NBA * NBA);
    double acc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k] = 0.0;
    if (inside(c, Jx, Jy, Jz)) {
      // per axis: slot of J in the P_s row of fine node x + d - RF (-1: none)
      int sx[W], sy[W], sz[W];
#pragma unroll
      for (int d = 0; d < W; ++d) {
        const int ix = x + d - RF, iy = y + d - RF, iz = z + d - RF;
        const int ax = Jx - ceil_half(ix - PR), ay = Jy - ceil_half(iy - PR), az = Jz - ceil_half(iz - PR);
        sx[d] = (ix >= 0 && ix <= f.lx && ax >= 0 && ax <= PR) ? ax : -1;
        sy[d] = (iy >= 0 && iy <= f.ly && ay >= 0 && ay <= PR) ? ay : -1;
        sz[d] = (iz >= 0 && iz <= f.lz && az >= 0 && az <= PR) ? az : -1;
      }
      const double* As = sA + nl * NB * 9;
#pragma unroll
      for (int dz = 0; dz < W; ++dz) {
        if (sz[dz] < 0) continue;
#pragma unroll
        for (int dy = 0; dy < W; ++dy) {
          if (sy[dy] < 0) continue;
#pragma unroll
          for (int dx = 0; dx < W; ++dx) {
            if (sx[dx] < 0) continue;
            const int q = p + (dx - RF) + f.px * ((dy - RF) + f.py * (dz - RF));
            const double* P = psb + (long long)q * NS * 9 + (sz[dz] * NA + sy[dy]) * NA + sx[dx];
            const double* A = As + ((dz * W + dy) * W + dx) * 9;
            double Pv[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) Pv[k] = __ldg(P + k * NS);
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
              for (int cc = 0; cc < 3; ++cc)
                acc[3 * r + cc] += A[3 * r] * Pv[cc] + A[3 * r + 1] * Pv[3 + cc] + A[3 * r + 2] * Pv[6 + cc];
          }
        }
      }
    }
    double* out = bsb + (long long)p * NSB * 9 + b;
#pragma unroll
    for (int k = 0; k < 9; ++k) out[k * NSB] = acc[k];
  }
}

// Lower offsets from the upper ones: block (s, p)[r][c] = block (NB-1-s, p + off(s))[c][r].
__global__ void k_wide_mirror(Grid c, int R, double* __restrict__ stc) {
  const int W = wide_w(R), NB = wide_nb(R), SC = NB / 2;
  const long long nint = (long long)(c.lx + 1) * (c.ly + 1) * (c.lz + 1);
  const long long nc = c.n;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)SC * nint;
       t += (long long)gridDim.x * blockDim.x) {
    const int s = (int)(t / nint);
    int X, Y, Z;
    interior_xyz(c, t % nint, X, Y, Z);
    const int p = c.idx(X, Y, Z);
    const int MX = X + s % W - R, MY = Y + (s / W) % W - R, MZ = Z + s / (W * W) - R;
    const bool in = inside(c, MX, MY, MZ);
    const long long q = in ? c.idx(MX, MY, MZ) : 0;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int cc = 0; cc < 3; ++cc)
        stc[((long long)s * 9 + 3 * r + cc) * nc + p] =
            in ? stc[((long long)(NB - 1 - s) * 9 + 3 * cc + r) * nc + q] : 0.0;
  }
}

// D_{l+1} from the diagonal, rows / columns of the other DOFs zeroed, Minv.
__global__ void k_wide_mask_from_diag(Grid c, int R, const double* __restrict__ st, uint8_t* __restrict__ cmask) {
  const int SC = wide_nb(R) / 2;
  const long long n = c.n;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < c.n; p += gridDim.x * blockDim.x) {
    int x, y, z;
    decode(c, p, x, y, z);
    uint8_t m = 0;
    if (inside(c, x, y, z))
      for (int r = 0; r < 3; ++r)
        if (st[((long long)SC * 9 + 4 * r) * n + p] > 0.0) m |= (uint8_t)(1 << r);
    cmask[p] = m;
  }
}

__global__ void k_wide_apply_mask(Grid c, int R, double* __restrict__ st, const uint8_t* __restrict__ cmask,
                                  double* __restrict__ minv3) {
  const int W = wide_w(R), NB = wide_nb(R), SC = NB / 2;
  const long long n = c.n;
  // one thread per node and block: a thread per node walked 125 blocks alone
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n * NB; i += (long long)gridDim.x * blockDim.x) {
    const int s = (int)(i / n), p = (int)(i - s * n);
    int x, y, z;
    decode(c, p, x, y, z);
    const bool in = inside(c, x, y, z);
    const uint8_t mp = cmask[p];
    {
      const int qx = x + s % W - R, qy = y + (s / W) % W - R, qz = z + s / (W * W) - R;
      const uint8_t mq = (in && inside(c, qx, qy, qz)) ? cmask[c.idx(qx, qy, qz)] : (uint8_t)0;
      for (int r = 0; r < 3; ++r)
        for (int cc = 0; cc < 3; ++cc)
          if (!(in && ((mp >> r) & 1) && ((mq >> cc) & 1))) st[((long long)s * 9 + 3 * r + cc) * n + p] = 0.0;
    }
    if (s == SC) for (int r = 0; r < 3; ++r) {
      const double d = st[((long long)SC * 9 + 4 * r) * n + p];
      minv3[3LL * p + r] = ((mp >> r) & 1) && d != 0.0 ? 1.0 / d : 0.0;
    }
  }
}

// ---- scaled symmetric storage ----------------------------------------------
template <typename S> __device__ __forceinline__ S to_s(double v);
template <> __device__ __forceinline__ float to_s<float>(double v) { return (float)v; }
template <> __device__ __forceinline__ double to_s<double>(double v) { return v; }
template <> __device__ __forceinline__ __half to_s<__half>(double v) { return __double2half(v); }

template <typename S, int R>
__global__ void k_wide_compress(Grid g, const double* __restrict__ st, const uint8_t* __restrict__ mask,
                                S* __restrict__ stc, typename WideLayout<S, R>::Q* __restrict__ sqrtd) {
  using L = WideLayout<S, R>;
  using Q = typename L::Q;
  constexpr int W = 2 * R + 1, NB = W * W * W, SC = NB / 2, G = L::G;
  const long long n = g.n;
  // one thread per node and block slot, a node's lanes consecutive (a thread
  // per node walked 64 slots alone: 0.27 ms on 2,400 nodes and on 20,000)
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n * G * L::NJ;
       i += (long long)gridDim.x * blockDim.x) {
    const int jj = (int)(i / (n * G)), p = (int)((i - jj * n * G) / G), u = jj * G + (int)(i % G);
    int x, y, z;
    decode(g, p, x, y, z);
    const bool in = inside(g, x, y, z);
    double sp[3];
    for (int r = 0; r < 3; ++r) {
      const double d = in ? st[((long long)SC * 9 + 4 * r) * n + p] : 0.0;
      sp[r] = (in && ((mask[p] >> r) & 1) && d > 0.0) ? 1.0 / sqrt(d) : 0.0;
      if (u == 0) sqrtd[3LL * p + r] = (Q)(sp[r] > 0.0 ? 1.0 / sp[r] : 0.0);
    }
    const long long v = (long long)p * G + u % G;
    if (jj == 0)
      for (int k = 9 * L::NJ; k < L::NVL; ++k) stc[L::off(v, k)] = to_s<S>(0.0);
    {
      const int k0 = 9 * (u / G);
      if (u >= L::NBLK) {
        for (int k = 0; k < 9; ++k) stc[L::off(v, k0 + k)] = to_s<S>(0.0);
        continue;
      }
      const int s = (u == L::NU) ? SC : SC + 1 + u;
      const int qx = x + s % W - R, qy = y + (s / W) % W - R, qz = z + s / (W * W) - R;
      double sq[3] = {0.0, 0.0, 0.0};
      if (in && inside(g, qx, qy, qz)) {
        const int q = g.idx(qx, qy, qz);
        for (int cc = 0; cc < 3; ++cc) {
          const double d = st[((long long)SC * 9 + 4 * cc) * n + q];
          sq[cc] = (((mask[q] >> cc) & 1) && d > 0.0) ? 1.0 / sqrt(d) : 0.0;
        }
      }
      for (int r = 0; r < 3; ++r)
        for (int cc = 0; cc < 3; ++cc) {
          const double val = (sp[r] != 0.0 && sq[cc] != 0.0) ? st[((long long)s * 9 + 3 * r + cc) * n + p] * sp[r] * sq[cc]
                                                             : 0.0;
          stc[L::off(v, k0 + 3 * r + cc)] = to_s<S>(val);
        }
    }
  }
}

// y = mask(D^1/2 A~ D^1/2 u) with the epilogues of the other level kernels
// (APPLY, SMOOTH with the Chebyshev step fields, RESID; a null rhs reads as
// zero; no fused dot product: the PCG's reductions run on level 0).  L::G
// lanes per node: each lane applies its own blocks and the transposed blocks
// of the same lane and slot of the lower neighbours, the partial sums meet
// through warp shuffles, and lanes 0..2 write component 0..2 of the node.
//
// A CTA owns 8 (reach 2) or 16 (reach 1) nodes of a row, one round of its 64
// threads: it stages v = D^1/2 u of them and their halo in shared memory with
// one set of loads, and the operator's loads depend on no branch, no table and
// not on u: the first batch is issued before anything else (RowBatch).  Bound
// by the latency of the loads on small levels and by the L1 on large ones.
// Against a form that walked the 8 block slots of a lane behind bounds tests
// and read u and the scale from global memory at every neighbour: 64x32x32
// part 185 -> 165 us an iteration, 96x80x64 315 -> 303, 128x64x64 FP64 534 ->
// 520, 256x128x128 1,401 -> 1,381.  The first batch ahead of the staging: 162 ->
// 153, 299 -> 286, 518 -> 507, 1,345 -> 1,333.  8 nodes a CTA instead of 16 on the
// reach-2 levels: 96x48x48 199 -> 189, 128x64x64 FP64 483 -> 466, others equal;
// larger tiles (32 x 1, 16 x 2 x 2, 16 x 4 x 4 nodes) and the slots split over
// 2 or 4 times the threads were slower or equal at every size.
template <typename T> struct Node3;   // 3 values of a node in shared memory
template <> struct Node3<float> {
  float4 v;
  __device__ __forceinline__ void get(float (&o)[3]) const { const float4 t = v; o[0] = t.x; o[1] = t.y; o[2] = t.z; }
  __device__ __forceinline__ void set(float a, float b, float c) { v = make_float4(a, b, c, 0.f); }
};
template <> struct Node3<double> {
  double v[3];
  __device__ __forceinline__ void get(double (&o)[3]) const { o[0] = v[0]; o[1] = v[1]; o[2] = v[2]; }
  __device__ __forceinline__ void set(double a, double b, double c) { v[0] = a; v[1] = b; v[2] = c; }
};
constexpr int wide_tx(int R) { return R == 1 ? 16 : 8; }   // nodes of a CTA

// f(integral constants I, I + STEP, ... < N)
template <int I, int N, int STEP, typename F> __device__ __forceinline__ void for_slots(F f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    for_slots<I + STEP, N, STEP>(f);
  }
}

template <typename T, typename S, int R, int EPI>
__global__ void __launch_bounds__(wide_tx(R) * WideLayout<S, R>::G)
    k_wide_op(Grid g, OpArgs a, const S* __restrict__ stc, const T* __restrict__ sqd) {
  pdl_enter();
  using L = WideLayout<S, R>;
  using A = T;
  constexpr int G = L::G, TX = wide_tx(R), HX = TX + 2 * R, HY = 1 + 2 * R, HZ = 1 + 2 * R, NT = TX * G;
  constexpr int JB = WideBatch<S>::JB;
  __shared__ Node3<T> sv[HX * HY * HZ];
  __shared__ int s_delta[G * L::NJ];
  KrylovState* ks = a.ks;
  const int done = ks ? ks->done : 0;
  const T* u = (const T*)a.u;
  T* out = (T*)a.out;
  const T* b = (const T*)a.b;
  const T* __restrict__ minv = (const T*)(EPI == EPI_APPLY ? a.apply_minv : a.minv);
  const T w = a.omega_dev ? (T)(*a.omega_dev) : (T)a.omega;
  const T* dprev = (const T*)a.dprev;
  T* dout = (T*)a.dout;
  const T c1 = a.c1_dev ? (T)(*a.c1_dev) : (T)0;
  const int ntx = (g.lx + TX) / TX;
  const int X0 = (blockIdx.x % ntx) * TX, y = blockIdx.x / ntx % (g.ly + 1), z = blockIdx.x / (ntx * (g.ly + 1));
  const int tx = threadIdx.x / G, lane = threadIdx.x % G, x = X0 + tx;
  const bool in = inside(g, x, y, z);
  const int p = in ? g.idx(x, y, z) : 0;
  RowBatch<S, L, JB> rb;
  rb.template load<0>(g, stc, p, lane);
  if (done) return;
  if (threadIdx.x < G * L::NJ) {
    constexpr int W = L::W, SC = L::NB / 2;
    const int uu = threadIdx.x, s = uu < L::NU ? SC + 1 + uu : SC;
    s_delta[uu] = ((s / (W * W) - R) * HY + (s / W) % W - R) * HX + s % W - R;
  }
  // halo nodes outside the grid read as zero, like the ghost shell
#pragma unroll
  for (int i0 = 0; i0 < HX * HY * HZ; i0 += NT) {
    const int i = i0 + threadIdx.x;
    const int hx = X0 - R + i % HX, hy = y - R + i / HX % HY, hz = z - R + i / (HX * HY);
    T v0 = 0, v1 = 0, v2 = 0;
    if (i < HX * HY * HZ && inside(g, hx, hy, hz)) {
      const long long q = 3LL * g.idx(hx, hy, hz);
      v0 = __ldg(sqd + q) * u[q];
      v1 = __ldg(sqd + q + 1) * u[q + 1];
      v2 = __ldg(sqd + q + 2) * u[q + 2];
    }
    if (i < HX * HY * HZ) sv[i].set(v0, v1, v2);
  }
  const int c = lane < 3 ? lane : 0;
  const long long pc = 3LL * p + c;
  T bc = 0, u0 = 0, mi = 0, dp = 0;
  const uint8_t m = __ldg(a.mask + p);
  const bool fr = (m >> c) & 1;
  const A sq = (A)__ldg(sqd + pc);
  if (lane < 3) {
    if (EPI != EPI_APPLY && b) bc = b[pc];
    if (EPI != EPI_RESID) u0 = u[pc];
    if (EPI != EPI_RESID && minv) mi = __ldg(minv + pc);
    if (EPI == EPI_SMOOTH && dprev) dp = dprev[pc];
  }
  __syncthreads();
  A acc[3] = {(A)0, (A)0, (A)0};
  const int c0 = (R * HY + R) * HX + tx + R;
  auto V = [&](int slot, A (&vu)[3], A (&vd)[3]) {
    const int d = s_delta[lane + G * slot];
    sv[c0 + d].get(vu);
    sv[c0 - d].get(vd);
  };
  rb.template apply<0>(lane, acc, V);
  for_slots<JB, L::NJ, JB>([&](auto j) {
    rb.template load<decltype(j)::value>(g, stc, p, lane);
    rb.template apply<decltype(j)::value>(lane, acc, V);
  });
#pragma unroll
  for (int o = 1; o < G; o <<= 1) {
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
  }
  if (!in || lane >= 3) return;
  const A ac = c == 0 ? acc[0] : (c == 1 ? acc[1] : acc[2]);
  const T kc = fr ? (T)(ac * sq) : (T)0;
  if (EPI == EPI_APPLY) {
    out[pc] = minv ? kc * mi : kc;
  } else if (EPI == EPI_SMOOTH) {
    T o = u0 + (fr ? w * (mi * (bc - kc)) : (T)0);
    if (dprev) o += c1 * dp;
    out[pc] = o;
    if (dout) dout[pc] = o - u0;
  } else {
    out[pc] = bc - kc;
  }
}

// Dense row-major A of a reach-R level (reference node order, DOF 3*node + c),
// identity rows on non-free DOFs.
__global__ void k_wide_dense_assemble(Grid c, int R, const double* __restrict__ st, const uint8_t* __restrict__ cm,
                                      double* __restrict__ A, int n) {
  const int W = wide_w(R), NB = wide_nb(R), SC = NB / 2;
  const int nx1 = c.lx + 1, ny1 = c.ly + 1;
  const long long nint = (long long)nx1 * ny1 * (c.lz + 1);
  const long long ns = c.n;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nint * NB;
       t += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(t / NB), s = (int)(t % NB);
    int x, y, z;
    interior_xyz(c, r, x, y, z);
    const int X = x + s % W - R, Y = y + (s / W) % W - R, Z = z + s / (W * W) - R;
    if (!inside(c, X, Y, Z)) continue;
    const int q = X + nx1 * (Y + ny1 * Z);
    const int p = c.idx(x, y, z);
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j)
        A[(long long)(3 * r + i) * n + 3 * q + j] = st[((long long)s * 9 + 3 * i + j) * ns + p];
    if (s == SC) {
      const uint8_t m = cm[p];
      for (int i = 0; i < 3; ++i)
        if (!((m >> i) & 1)) A[(long long)(3 * r + i) * n + 3 * r + i] = 1.0;
    }
  }
}

__global__ void k_smoothing_coef(const double* __restrict__ lambda, double* __restrict__ coef) {
  const double l = *lambda;
  *coef = l > 0.0 ? (4.0 / 3.0) / l : 0.0;
}

}  // namespace

// ---- launchers ---------------------------------------------------------------
void launch_smoothing_coef(const double* lambda, double* coef, cudaStream_t st) {
  launch_k(k_smoothing_coef, 1, 1, 0, st, lambda, coef);
}

size_t wide_prolong_count(const Grid& f, int Pr) { return (size_t)f.n * (Pr + 1) * (Pr + 1) * (Pr + 1) * 9; }
size_t wide_rapb_count(const Grid& f, int Pr, int Rf) {
  const size_t a = (size_t)(Pr + Rf + 1);
  return (size_t)f.n * a * a * a * 9;
}

void launch_wide_galerkin(const Grid& f, const double* stf, int Rf, const uint8_t* fmask, const double* minvf,
                          const double* cdev, int Pr, const Grid& c, double* stc, int Rc, double* psb, double* bsb,
                          cudaStream_t st) {
  const long long nintf = (long long)(f.lx + 1) * (f.ly + 1) * (f.lz + 1);
  const long long nintc = (long long)(c.lx + 1) * (c.ly + 1) * (c.lz + 1);
  const int NS = (Pr + 1) * (Pr + 1) * (Pr + 1), NBA = Pr + Rf + 1, NSB = NBA * NBA * NBA;
  const int ngp = kSetupThreads / NS, ngb = kSetupThreads / NSB;
  const int gp = (int)std::min<long long>((nintf + ngp - 1) / ngp, 148LL * 64);
  const int gb = (int)std::min<long long>((nintf + ngb - 1) / ngb, 148LL * 64);
  const int gc = (int)std::min<long long>(nintc, 148LL * 256);
  const size_t smem_c = sizeof(double) * (2 * Pr + 1) * (2 * Pr + 1) * (2 * Pr + 1) * 9;   // k_rap_c
  // the two pairs the hierarchy builds (see k_prolong_blocks_t)
#define VF_WIDE_FIXED(RF_, PR_, SM_)                                                                          \
  do {                                                                                                        \
    launch_k(k_prolong_blocks_t<RF_, PR_, SM_>, gp, kSetupThreads, 0, st, f, stf, fmask, minvf, cdev, c, psb); \
    launch_k(k_rap_b_t<RF_, PR_>, gb, kSetupThreads, 0, st, f, stf, (const double*)psb, c, bsb);             \
    launch_k(k_rap_c, gc, kRapThreads, smem_c, st, f, Rf, (const double*)psb, Pr, (const double*)bsb, c, Rc, stc); \
    launch_k(k_wide_mirror, blocks_for((long long)(wide_nb(Rc) / 2) * nintc, 128), 128, 0, st, c, Rc, stc);    \
    return;                                                                                                   \
  } while (0)
  if (Rf == 1 && Pr == 2 && Rc == 2 && cdev) VF_WIDE_FIXED(1, 2, true);
  if (Rf == 2 && Pr == 1 && Rc == 2 && !cdev) VF_WIDE_FIXED(2, 1, false);
#undef VF_WIDE_FIXED
  const size_t smem_p = cdev ? sizeof(double) * ngp * wide_nb(Rf) * 9 : 0;
  const size_t smem_b = sizeof(double) * ngb * wide_nb(Rf) * 9;
  launch_k(k_prolong_blocks, (int)std::min<long long>((nintf + ngp - 1) / ngp, 148LL * 64), kSetupThreads, smem_p, st,
           f, stf, Rf, fmask, minvf, cdev, Pr, c, psb);
  launch_k(k_rap_b, (int)std::min<long long>((nintf + ngb - 1) / ngb, 148LL * 64), kSetupThreads, smem_b, st, f, stf,
           Rf, psb, Pr, c, bsb);
  const int WI = 2 * Pr + 1;
  const size_t smem = sizeof(double) * WI * WI * WI * 9;
  launch_k(k_rap_c, (int)std::min<long long>(nintc, 148LL * 256), kRapThreads, smem, st, f, Rf, psb, Pr, bsb, c, Rc,
           stc);
  launch_k(k_wide_mirror, blocks_for((long long)(wide_nb(Rc) / 2) * nintc, 128), 128, 0, st, c, Rc, stc);
}

void launch_wide_mask(const Grid& c, int R, double* stc, uint8_t* cmask, double* minv3, cudaStream_t st) {
  launch_k(k_wide_mask_from_diag, blocks_for(c.n, 256), 256, 0, st, c, R, stc, cmask);
  launch_k(k_wide_apply_mask, blocks_for((long long)c.n * wide_nb(R), 128), 128, 0, st, c, R, stc, cmask, minv3);
}

template <typename S, int R>
void launch_wide_compress(const Grid& g, const double* st, const uint8_t* mask, S* stc,
                          typename WideLayout<S, R>::Q* sqrtd, cudaStream_t st_) {
  launch_k(k_wide_compress<S, R>, blocks_for((long long)g.n * WideLayout<S, R>::G * WideLayout<S, R>::NJ, 128), 128, 0, st_, g, st, mask, stc, sqrtd);
}

template <typename T, typename S, int R>
void launch_wide_op(const Grid& g, int epi, const OpArgs& a, const S* stc, const T* sqrtd, bool early, cudaStream_t st) {
  constexpr int TX = wide_tx(R), NT = TX * WideLayout<S, R>::G;
  const unsigned blocks = (unsigned)((g.lx + TX) / TX) * (g.ly + 1) * (g.lz + 1);
  auto go = [&](auto kern) {
    if (early) launch_pdl(kern, blocks, NT, 0, st, g, a, stc, sqrtd);
    else launch_k(kern, blocks, NT, 0, st, g, a, stc, sqrtd);
  };
  if (epi == EPI_APPLY) go(k_wide_op<T, S, R, EPI_APPLY>);
  else if (epi == EPI_SMOOTH) go(k_wide_op<T, S, R, EPI_SMOOTH>);
  else go(k_wide_op<T, S, R, EPI_RESID>);
}
#define VF_INST_WIDE(T, S)                                                                                          \
  template void launch_wide_op<T, S, 1>(const Grid&, int, const OpArgs&, const S*, const T*, bool, cudaStream_t);   \
  template void launch_wide_op<T, S, 2>(const Grid&, int, const OpArgs&, const S*, const T*, bool, cudaStream_t);   \
  template void launch_wide_compress<S, 1>(const Grid&, const double*, const uint8_t*, S*, T*, cudaStream_t);       \
  template void launch_wide_compress<S, 2>(const Grid&, const double*, const uint8_t*, S*, T*, cudaStream_t);
VF_INST_WIDE(float, __half)
VF_INST_WIDE(float, float)
VF_INST_WIDE(double, double)
#undef VF_INST_WIDE

int wide_dense_assemble(const Grid& c, int R, const double* stencil, const uint8_t* cmask, double* A, int n,
                        cudaStream_t st) {
  cudaMemsetAsync(A, 0, sizeof(double) * (size_t)n * n, st);
  const long long work = (long long)(c.lx + 1) * (c.ly + 1) * (c.lz + 1) * wide_nb(R);
  launch_k(k_wide_dense_assemble, blocks_for(work, 256, 148LL * 256), 256, 0, st, c, R, stencil, cmask, A, n);
  return 0;
}

}  // namespace vf
