// The reference's coarsest "solve" (core/multigrid.py:428-429: 30 damped-Jacobi
// sweeps from zero) in one launch, for element-operator levels small enough to
// live in one SM's shared memory.
//
// On a coarsest level of a few hundred nodes a sweep is a microsecond of
// arithmetic; as a launch of its own it cost 4.3 us in a graph, 29 of them in
// each V-cycle (the 64x16x16 beam, 16x4x4 coarsest level: 2.5 of 5 ms).  Here
// one block keeps the iterate, the right-hand side and the weighted inverse
// diagonal in shared memory and alternates two phases: a thread per element
// transforms its 24 corner values to modes (vf_modal.cuh) and leaves its corner
// forces in shared memory, a thread per node sums its elements' forces and
// updates.  One block, not a cluster: the level has less work than a cluster's
// barrier and its trips to L2 cost (16 blocks: 3.8 us a sweep).
#include <atomic>

#include "vf_common.cuh"
#include "vf_modal.cuh"

namespace vf {

namespace modal {
template <> __device__ __forceinline__ float bc<float>(double v) { return (float)v; }
}  // namespace modal

namespace {

constexpr int kCoarseThreads = 512;

template <typename T> struct Scalar {
  using P = T;
  __device__ __forceinline__ static T add(T a, T b) { return a + b; }
  __device__ __forceinline__ static T sub(T a, T b) { return a - b; }
  __device__ __forceinline__ static T mul(T a, T b) { return a * b; }
  __device__ __forceinline__ static T fma(T a, T b, T c) { return ::fma(a, b, c); }
};

// values in shared memory: u, b and w Minv (3 per node), forces (24 per element)
size_t coarse_values(const Grid& g) { return 9 * (size_t)g.nodes_ref() + 24 * (size_t)g.elems_ref(); }

template <typename T, bool LAME>
__global__ void __launch_bounds__(kCoarseThreads, 1)
    k_coarse_jacobi(Grid g, const T* b, T* __restrict__ x, const T* __restrict__ minv,
                    const uint8_t* __restrict__ mask, const T* __restrict__ E, const T* __restrict__ MU, ModalConst mc,
                    int sweeps, T w0, const double* wdev, const KrylovState* ks) {
  pdl_enter();
  if (ks && ks->done) return;
  using O = Scalar<T>;
  extern __shared__ double smem[];
  const int nx1 = g.lx + 1, ny1 = g.ly + 1, nn = g.nodes_ref(), ne = g.elems_ref();
  T* u = reinterpret_cast<T*>(smem);
  T* sb = u + 3 * nn;
  T* sm = sb + 3 * nn;
  T* F = sm + 3 * nn;   // [corner][component][element]
  const T w = wdev ? (T)(*wdev) : w0;
  for (int i = threadIdx.x; i < 3 * nn; i += kCoarseThreads) {
    const int t = i / 3, c = i - 3 * t, r = t / nx1;
    const int p = g.idx(t % nx1, r % ny1, r / ny1);
    const bool fr = (mask[p] >> c) & 1;
    const T bi = b[3 * p + c], m = fr ? minv[3 * p + c] : (T)0;
    sb[i] = bi;
    sm[i] = m;
    u[i] = w * (m * bi);   // the first sweep, from zero
  }
  __syncthreads();
#pragma unroll 1
  for (int k = 1; k < sweeps; ++k) {
#pragma unroll 1
    for (int e = threadIdx.x; e < ne; e += kCoarseThreads) {
      const int r = e / g.lx, ex = e - r * g.lx, ey = r % g.ly, ez = r / g.ly;
      const T* q = u + 3 * (ex + nx1 * (ey + ny1 * ez));
      const int q0 = g.idx(ex, ey, ez);
      const T El = __ldg(E + q0), Em = LAME ? __ldg(MU + q0) : El;
      T A[3][8], B[3][8];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T f[2][4];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const T* qz = q + 3 * nx1 * ny1 * z + c;
          const T u00 = qz[0], u10 = qz[3], u01 = qz[3 * nx1], u11 = qz[3 * nx1 + 3];
          const T e0 = u10 + u00, e1 = u10 - u00, e2 = u11 + u01, e3 = u11 - u01;
          f[z][0] = e0 + e2; f[z][1] = e1 + e3; f[z][2] = e2 - e0; f[z][3] = e3 - e1;
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          A[c][m] = f[0][m] + f[1][m];
          A[c][m + 4] = f[1][m] - f[0][m];
        }
      }
      modal::modal_physics<O, T, T>(A, B, El, Em, mc);
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          T a[4];
          a[0] = z ? B[c][4] : -B[c][4];
#pragma unroll
          for (int m = 1; m < 4; ++m) a[m] = z ? B[c][m] + B[c][m + 4] : B[c][m] - B[c][m + 4];
          const T t0 = a[0] - a[2], t1 = a[1] - a[3], t2 = a[0] + a[2], t3 = a[1] + a[3];
          T* f = F + (size_t)(12 * z + c) * ne + e;   // corner 4 z + 2 y + x
          f[0] = t0 - t1;
          f[(size_t)3 * ne] = t0 + t1;
          f[(size_t)6 * ne] = t2 - t3;
          f[(size_t)9 * ne] = t2 + t3;
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int t = threadIdx.x; t < nn; t += kCoarseThreads) {
      const int r = t / nx1, nx = t - r * nx1, ny = r % ny1, nz = r / ny1;
      T s[3] = {0, 0, 0};
#pragma unroll
      for (int k8 = 0; k8 < 8; ++k8) {
        const int ex = nx - (k8 & 1), ey = ny - ((k8 >> 1) & 1), ez = nz - (k8 >> 2);
        if (ex < 0 || ex >= g.lx || ey < 0 || ey >= g.ly || ez < 0 || ez >= g.lz) continue;
        const T* f = F + (size_t)(3 * k8) * ne + ex + g.lx * (ey + g.ly * ez);
        s[0] += f[0]; s[1] += f[ne]; s[2] += f[(size_t)2 * ne];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) u[3 * t + c] += w * (sm[3 * t + c] * (sb[3 * t + c] - s[c]));
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < 3 * nn; i += kCoarseThreads) {
    const int t = i / 3, c = i - 3 * t, r = t / nx1;
    x[3 * g.idx(t % nx1, r % ny1, r / ny1) + c] = u[i];
  }
}

constexpr size_t kCoarseSmem = 220 * 1024;

}  // namespace

template <typename T>
bool launch_coarse_jacobi(const Grid& g, const T* b, T* x, const T* minv3, const uint8_t* mask, const T* E, const T* mu,
                          const ModalConst& mc, int sweeps, double omega, const double* omega_dev,
                          const KrylovState* ks, cudaStream_t st) {
  const size_t smem = sizeof(T) * coarse_values(g);
  if (sweeps < 2 || smem > kCoarseSmem) return false;
  static std::atomic<int> per_dev[2][kMaxDevices];
  if (mu) {
    kernel_prepare(per_dev[0], k_coarse_jacobi<T, true>, kCoarseSmem, kCoarseThreads);
    launch_pdl(k_coarse_jacobi<T, true>, 1, kCoarseThreads, smem, st, g, b, x, minv3, mask, E, mu, mc, sweeps, (T)omega,
               omega_dev, ks);
  } else {
    kernel_prepare(per_dev[1], k_coarse_jacobi<T, false>, kCoarseSmem, kCoarseThreads);
    launch_pdl(k_coarse_jacobi<T, false>, 1, kCoarseThreads, smem, st, g, b, x, minv3, mask, E, mu, mc, sweeps,
               (T)omega, omega_dev, ks);
  }
  return true;
}
template bool launch_coarse_jacobi<float>(const Grid&, const float*, float*, const float*, const uint8_t*, const float*,
                                          const float*, const ModalConst&, int, double, const double*,
                                          const KrylovState*, cudaStream_t);
template bool launch_coarse_jacobi<double>(const Grid&, const double*, double*, const double*, const uint8_t*,
                                           const double*, const double*, const ModalConst&, int, double, const double*,
                                           const KrylovState*, cudaStream_t);

}  // namespace vf
