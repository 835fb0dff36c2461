// Coarsest-level direct solve in FP64: the assembled coarsest operator (with
// identity rows on non-free DOFs) is factored A = L L^T by a blocked
// right-looking Cholesky, inverted as A^{-1} = Y^T Y with Y = L^{-1}, and each
// V-cycle applies the explicit inverse with one GEMV.  All kernels are plain
// CUDA-core FP64; the factorization runs once per set_material, outside the
// iteration.  A coarsest level of many DOFs (a grid that halves only once or
// twice) is dissected instead: see DensePlan below.
// Replaces the reference's 30-sweep Jacobi "coarse solve" (core/multigrid.py:428-429)
// when VF_COARSEST_CHOLESKY is selected.
#include <algorithm>

#include "vf_common.cuh"

namespace vf {

namespace {

constexpr int NB = 32;

// Dense row-major A from the coarsest stencil; node order = reference order
// of the level's nodes, DOF 3*node + c.
__global__ void k_dense_assemble(Grid c, const double* __restrict__ st, const uint8_t* __restrict__ cm,
                                 double* __restrict__ A, int n) {
  const int nx1 = c.lx + 1, ny1 = c.ly + 1, nint = nx1 * ny1 * (c.lz + 1);
  const long long ns = c.n;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nint * 27; t += gridDim.x * blockDim.x) {
    const int r = t / 27, s = t % 27;
    const int x = r % nx1, rr = r / nx1, y = rr % ny1, z = rr / ny1;
    const int dx = s % 3 - 1, dy = (s / 3) % 3 - 1, dz = s / 9 - 1;
    const int X = x + dx, Y = y + dy, Z = z + dz;
    if (X < 0 || X > c.lx || Y < 0 || Y > c.ly || Z < 0 || Z > c.lz) continue;
    const int q = X + nx1 * (Y + ny1 * Z);
    const int p = c.idx(x, y, z);
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b)
        A[(long long)(3 * r + a) * n + 3 * q + b] = st[((long long)s * 9 + a * 3 + b) * ns + p];
    if (s == 13) {
      const uint8_t m = cm[p];
      for (int a = 0; a < 3; ++a)
        if (!((m >> a) & 1)) A[(long long)(3 * r + a) * n + 3 * r + a] = 1.0;
    }
  }
}

// Factor the nb x nb diagonal block at (k, k) (rows already updated) and
// invert it: L_kk -> A's lower block, L_kk^-1 -> linv (NB x NB, zero padded).
// 1024 threads, one per (row t, column c) of the block; the panel solve and
// the block-row solve of the inverse phase then multiply by linv instead of
// substituting row by row.
// (blockIdx.x: matrix of a batch, sA / sL values apart.  info: the least of
// row0 + n * matrix + row over the rows whose pivot was not positive.)
__global__ void __launch_bounds__(NB * NB, 1) k_potrf_diag(double* A, int n, int k, int nb, int* info, double* linv,
                                                           size_t sA, size_t sL, int row0) {
  pdl_enter();
  A += sA * blockIdx.x;
  linv += sL * blockIdx.x;
  // L: the block being reduced (column j is read, columns > j updated in step
  // j); F: the factor, each entry written once -- so one barrier per column:
  // every thread takes the pivot's square root itself, and nothing reads
  // what step j writes until step j + 1
  __shared__ double L[NB][NB + 1], F[NB][NB + 1], X[NB][NB + 1], rec[NB];
  const int c = threadIdx.x % NB, t = threadIdx.x / NB;
  L[t][c] = (t < nb && c <= t) ? A[(long long)(k + t) * n + k + c] : 0.0;
  F[t][c] = 0.0;
  __syncthreads();
  for (int j = 0; j < nb; ++j) {
    const double d = L[j][j];
    const bool bad = !(d > 0.0);
    const double piv = bad ? 1.0 : sqrt(d);
    const double rinv = 1.0 / piv;
    if (t == j && c == j) {
      F[j][j] = piv;
      rec[j] = rinv;
      if (bad) atomicMin(info, row0 + n * (int)blockIdx.x + k + j);
    }
    if (t > j && t < nb) {
      const double lt = L[t][j] * rinv;
      if (c == j) F[t][j] = lt;
      else if (c > j && c <= t) L[t][c] -= lt * (L[c][j] * rinv);
    }
    __syncthreads();
  }
  // X = F^-1 by right-looking substitution: thread (t, c) keeps X[t][c] in a
  // register; step r finalises row r and every lower row subtracts its
  // multiple of it -- one FMA and one barrier per step
  double xv = (t == c) ? 1.0 : 0.0;
  for (int r = 0; r < nb; ++r) {
    if (t == r) {
      xv *= rec[r];   // (a division here was a third of the kernel's chain)
      X[r][c] = xv;
    }
    __syncthreads();
    if (t > r && t < nb) xv = fma(-F[t][r], X[r][c], xv);
  }
  if (t < nb && c <= t) A[(long long)(k + t) * n + k + c] = F[t][c];
  linv[t * NB + c] = (t < nb && c < nb) ? X[t][c] : 0.0;
}

// Rows i >= k+nb: A[i, k:k+nb] <- A[i, k:k+nb] L_kk^-T, i.e.
// X[i][j] = sum_{l <= j} A[i][k+l] linv[j][l].  64 rows per CTA.
__global__ void __launch_bounds__(256) k_trsm_panel(double* A, int n, int k, int nb, const double* linv, size_t sA,
                                                    size_t sL) {
  pdl_enter();
  A += sA * blockIdx.y;
  linv += sL * blockIdx.y;
  __shared__ double P[64][NB + 1], Li[NB][NB + 1];
  const int tid = threadIdx.x;
  const int i0 = k + nb + blockIdx.x * 64;
  for (int e = tid; e < NB * NB; e += 256) Li[e / NB][e % NB] = linv[e];
  for (int e = tid; e < 64 * NB; e += 256) {
    const int r = e / NB, l = e % NB;
    P[r][l] = (i0 + r < n && l < nb) ? A[(long long)(i0 + r) * n + k + l] : 0.0;
  }
  __syncthreads();
  const int c = tid % NB, r0 = tid / NB;
  for (int a = 0; a < 8; ++a) {
    const int r = r0 + 8 * a;
    double v = 0.0;
    for (int l = 0; l <= c; ++l) v = fma(P[r][l], Li[c][l], v);
    if (i0 + r < n && c < nb) A[(long long)(i0 + r) * n + k + c] = v;
  }
}

// The three O(n^3) phases (trailing update, the update of Y = L^-1, Y^T Y)
// run on 64 x 64 output tiles per CTA of 256 threads, each thread holding a
// 4 x 4 register block (rows ty + 16a, columns tx + 16b): per inner index one
// shared-memory load of 4 + 4 values feeds 16 FMAs.
constexpr int TB = 64;

// Trailing update (lower triangle): A[i][j] -= sum_l A[i][k+l] A[j][k+l].
// Grid: one CTA per 64 x 64 tile pair bi >= bj of the trailing matrix.
__global__ void __launch_bounds__(256) k_syrk_update(double* A, int n, int k, int nb, size_t sA) {
  pdl_enter();
  A += sA * blockIdx.z;
  const int t0 = k + nb;
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  const int i0 = t0 + bi * TB, j0 = t0 + bj * TB;
  __shared__ double Pi[TB][NB + 1], Pj[TB][NB + 1];
  const int tid = threadIdx.x;
  for (int e = tid; e < TB * NB; e += 256) {
    const int r = e / NB, l = e % NB;
    Pi[r][l] = (i0 + r < n && l < nb) ? A[(long long)(i0 + r) * n + k + l] : 0.0;
    Pj[r][l] = (j0 + r < n && l < nb) ? A[(long long)(j0 + r) * n + k + l] : 0.0;
  }
  __syncthreads();
  const int tx = tid % 16, ty = tid / 16;
  double acc[4][4] = {};
  for (int l = 0; l < nb; ++l) {
    double pi[4], pj[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) pi[a] = Pi[ty + 16 * a][l];
#pragma unroll
    for (int b = 0; b < 4; ++b) pj[b] = Pj[tx + 16 * b][l];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = fma(pi[a], pj[b], acc[a][b]);
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
      if (i < n && j <= i) A[(long long)i * n + j] -= acc[a][b];
    }
}

// Y = L^-1 by recursive doubling over the 32-row block structure (the
// blocked triangular inversion): with both halves of a block pair already
// inverted,
//     [L11 0; L21 L22]^-1 = [Y11 0; -Y22 L21 Y11  Y22],
// so each level is two batched products over all pairs of the level:
// T = L21 Y11, then Y21 = -Y22 T.  8 levels for n = 4,131 (16 launches
// instead of a 130-step substitution whose products had K = 32).
struct GemmJob {
  const double* A; const double* B; double* C;   // C (M x N) = alpha A (M x K) B (K x N), row-major
  int lda, ldb, ldc, M, N, K;
};
constexpr int kMaxJobs = 128;
struct GemmBatch {
  GemmJob job[kMaxJobs];
  int count;
  double alpha, beta;     // C = alpha A B + beta C (C is not read when beta is 0)
  int a_lower, b_lower;   // A / B lower triangular (square): skip the zero part of the K range
  // a_bw > 0: A is a block L21 of a band matrix, its row 0 K rows below its
  // column 0, so A[i][k] = 0 for k < i + K - a_bw
  int a_bw;
};

// One 64 x 64 output tile per CTA (blockIdx.x: tile of job blockIdx.y),
// 4 x 4 register blocks, K in chunks of 32 through shared memory.
__global__ void __launch_bounds__(256) k_gemm_batched(const __grid_constant__ GemmBatch bt) {
  pdl_enter();
  const GemmJob& jb = bt.job[blockIdx.y];
  const int tn = (jb.N + TB - 1) / TB, tm = (jb.M + TB - 1) / TB;
  if ((int)blockIdx.x >= tn * tm) return;
  const int i0 = ((int)blockIdx.x / tn) * TB, j0 = ((int)blockIdx.x % tn) * TB;
  int kb = 0, ke = jb.K;
  if (bt.b_lower) kb = j0;                        // B[k][j] = 0 for k < j
  if (bt.a_lower) ke = min(ke, i0 + TB);          // A[i][k] = 0 for k > i
  if (bt.a_bw > 0) kb = max(kb, i0 + jb.K - bt.a_bw);
  constexpr int LC = 32;
  __shared__ double As[TB][LC + 1], Bs[LC][TB + 1];
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  double acc[4][4] = {};
  for (int k0 = kb; k0 < ke; k0 += LC) {
    for (int e = tid; e < TB * LC; e += 256) {
      const int r = e / LC, l = e % LC;
      const int gi = i0 + r, gk = k0 + l;
      As[r][l] = (gi < jb.M && gk < ke) ? jb.A[(long long)gi * jb.lda + gk] : 0.0;
      const int lr = e / TB, c = e % TB;
      const int gk2 = k0 + lr, gj = j0 + c;
      Bs[lr][c] = (gk2 < ke && gj < jb.N) ? jb.B[(long long)gk2 * jb.ldb + gj] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int l = 0; l < LC; ++l) {
      double a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = As[ty + 16 * q][l];
#pragma unroll
      for (int q = 0; q < 4; ++q) b[q] = Bs[l][tx + 16 * q];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int w = 0; w < 4; ++w) acc[q][w] = fma(a[q], b[w], acc[q][w]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int i = i0 + ty + 16 * q, j = j0 + tx + 16 * w;
      if (i < jb.M && j < jb.N) {
        double* C = jb.C + (long long)i * jb.ldc + j;
        *C = bt.beta != 0.0 ? bt.alpha * acc[q][w] + bt.beta * *C : bt.alpha * acc[q][w];
      }
    }
}

// Y = 0 with the inverted diagonal blocks L_kk^-1 on the diagonal.
__global__ void k_y_init(double* Y, int n, const double* linv_all, size_t sY, size_t sL) {
  Y += sY * blockIdx.y;
  linv_all += sL * blockIdx.y;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)n * n;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / n), j = (int)(e % n);
    double v = 0.0;
    if (i / NB == j / NB) {
      const int k = i / NB;
      v = linv_all[(size_t)k * NB * NB + (i - k * NB) * NB + (j - k * NB)];
    }
    Y[e] = v;
  }
}

// Ainv = Y^T Y (Y lower triangular): Ainv[i][j] = sum_{l >= max(i,j)} Y[l][i] Y[l][j].
// A^-1 = Y^T Y is symmetric: one CTA per 64x64 tile of the lower triangle
// (blockIdx.x enumerates the pairs bi >= bj), written to both triangles.
__global__ void __launch_bounds__(256) k_yty(const double* Y, double* Ainv, int n, size_t sY, size_t sA) {
  pdl_enter();
  Y += sY * blockIdx.y;
  Ainv += sA * blockIdx.y;
  int bi = (int)((sqrt(8.0 * blockIdx.x + 1.0) - 1.0) * 0.5);
  while ((bi + 1) * (bi + 2) / 2 <= (int)blockIdx.x) ++bi;
  while (bi * (bi + 1) / 2 > (int)blockIdx.x) --bi;
  const int bj = (int)blockIdx.x - bi * (bi + 1) / 2;
  const int i0 = bi * TB, j0 = bj * TB;
  constexpr int LC = 32;   // inner-index chunk
  __shared__ double Yi[LC][TB + 1], Yj[LC][TB + 1];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  double acc[4][4] = {};
  const int lstart = (i0 > j0 ? i0 : j0);
  for (int l0 = lstart; l0 < n; l0 += LC) {
    for (int e = tid; e < LC * TB; e += 256) {
      const int r = e / TB, c = e % TB;
      const int l = l0 + r;
      Yi[r][c] = (l < n && i0 + c < n) ? Y[(long long)l * n + i0 + c] : 0.0;
      Yj[r][c] = (l < n && j0 + c < n) ? Y[(long long)l * n + j0 + c] : 0.0;
    }
    __syncthreads();
    for (int l = 0; l < LC; ++l) {
      double yi[4], yj[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) yi[a] = Yi[l][ty + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) yj[b] = Yj[l][tx + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fma(yi[a], yj[b], acc[a][b]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
      if (i < n && j < n) {
        Ainv[(long long)i * n + j] = acc[a][b];
        Ainv[(long long)j * n + i] = acc[a][b];
      }
    }
}

// Padded-storage vector index of each coarsest DOF (reference node order,
// DOF 3 * node + c): the GEMVs gather b and scatter x through it instead of
// decoding node coordinates in every CTA.
__global__ void k_dense_perm(Grid c, int* __restrict__ perm, int n) {
  const int nx1 = c.lx + 1, ny1 = c.ly + 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int r = i / 3, comp = i - 3 * r;
    const int xx = r % nx1, rr = r / nx1, yy = rr % ny1, zz = rr / ny1;
    perm[i] = 3 * c.idx(xx, yy, zz) + comp;
  }
}

// FP32 copy of the FP64 inverse with rows padded to ld (a multiple of 4)
// floats, the padding zero: every row starts on a 16-byte boundary.
__global__ void k_convert_pad(const double* __restrict__ A, float* __restrict__ B, int n, int ld) {
  const long long total = (long long)n * ld;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / ld), j = (int)(e - (long long)i * ld);
    B[e] = j < n ? (float)A[(long long)i * n + j] : 0.0f;
  }
}

// x = Ainv b on the coarsest level; b gathered into shared memory in FP64,
// products accumulated in FP64 (Ainv in FP64; the FP32 V-cycle reads the
// padded FP32 copy in k_dense_solve_f32).
__global__ void k_dense_solve(const double* __restrict__ Ainv, int n, const int* __restrict__ perm, const double* b,
                              double* __restrict__ x, const KrylovState* ks) {
  pdl_enter();
  if (ks && ks->done) return;
  extern __shared__ double sb[];
  for (int i = threadIdx.x; i < n; i += blockDim.x) sb[i] = b[__ldg(perm + i)];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (int i = blockIdx.x * wpb + warp; i < n; i += gridDim.x * wpb) {
    const double* row = Ainv + (long long)i * n;
    // eight independent partial sums keep eight 256-byte row segments in
    // flight per warp (the GEMV streams n^2 doubles per call)
    double part[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int j = lane;
    for (; j + 7 * 32 < n; j += 8 * 32) {
#pragma unroll
      for (int k = 0; k < 8; ++k) part[k] += __ldg(row + j + 32 * k) * sb[j + 32 * k];
    }
    for (; j < n; j += 32) part[7] += __ldg(row + j) * sb[j];
    double s = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) x[__ldg(perm + i)] = s;
  }
}

// The FP32 V-cycle's coarsest GEMV: rows of ld floats (16-byte aligned,
// zero-padded past n), each lane streaming float4s, eight in flight per lane
// (4 KB per warp: enough bytes in flight to approach the HBM rate with one
// row per warp), products accumulated in FP64.
__global__ void k_dense_solve_f32(const float* __restrict__ Ainv, int n, int ld, const int* __restrict__ perm,
                                  const float* b, float* __restrict__ x, const KrylovState* ks) {
  pdl_enter();
  if (ks && ks->done) return;
  extern __shared__ double sb[];   // ld values, zero past n
  for (int i = threadIdx.x; i < ld; i += blockDim.x) sb[i] = i < n ? (double)b[__ldg(perm + i)] : 0.0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const int n4 = ld >> 2;
  for (int i = blockIdx.x * wpb + warp; i < n; i += gridDim.x * wpb) {
    const float4* row = reinterpret_cast<const float4*>(Ainv + (long long)i * ld);
    double part[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int j = lane;
    for (; j + 7 * 32 < n4; j += 8 * 32) {
      float4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __ldg(row + j + 32 * k);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double* bb = sb + 4 * (j + 32 * k);
        part[k] += (double)v[k].x * bb[0] + (double)v[k].y * bb[1] + (double)v[k].z * bb[2] +
                   (double)v[k].w * bb[3];
      }
    }
    for (; j < n4; j += 32) {
      const float4 v = __ldg(row + j);
      const double* bb = sb + 4 * j;
      part[7] += (double)v.x * bb[0] + (double)v.y * bb[1] + (double)v.z * bb[2] + (double)v.w * bb[3];
    }
    double s = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) x[__ldg(perm + i)] = (float)s;
  }
}

}  // namespace

int dense_assemble(const Grid& c, const double* stencil, const uint8_t* cmask, double* A, int n, cudaStream_t st) {
  cudaMemsetAsync(A, 0, sizeof(double) * (size_t)n * n, st);
  const long long work = (long long)(c.lx + 1) * (c.ly + 1) * (c.lz + 1) * 27;
  int blocks = (int)((work + 255) / 256);
  launch_k(k_dense_assemble, blocks, 256, 0, st, c, stencil, cmask, A, n);
  return 0;
}

// Doubles of the work buffer for a batch of n x n matrices: each Y = L^-1, its
// inverted diagonal blocks (NB x NB each) and the products' temporaries.
static size_t cholesky_work(int n, int batch) {
  return (size_t)batch * ((size_t)n * n + (size_t)((n + NB - 1) / NB) * NB * NB + (size_t)n * n / 2 + (size_t)NB * n);
}

// A (batch matrices n x n, sA values apart, lower parts) is overwritten by L;
// work (cholesky_work) receives Y = L^-1 and the inverted diagonal blocks;
// A <- Y^T Y = A^-1.  d_info receives the first row without a positive pivot,
// row0 + n * matrix + row, where it is below d_info's value.  bw: A[i][j] == 0
// for |i - j| > bw (a stencil operator in lexicographic node order is banded).
// A Cholesky factor keeps the band, so the panel solve and the trailing update
// of block column k only touch the rows below it that lie within the band: the
// rows they skip would receive exact zeros (the factor is the same bit for
// bit).
static void cholesky_inverse(double* A, double* work, int n, int bw, int* d_info, cudaStream_t st, int batch,
                             size_t sA, int row0) {
  const int nbk = (n + NB - 1) / NB;
  const size_t sY = (size_t)n * n, sL = (size_t)nbk * NB * NB;
  double* linv_all = work + sY * batch;
  if (bw < 0 || bw > n) bw = n;
  for (int k = 0; k < n; k += NB) {
    const int nb = (n - k < NB) ? (n - k) : NB;
    double* linv = linv_all + (size_t)(k / NB) * NB * NB;
    launch_pdl(k_potrf_diag, batch, NB * NB, 0, st, A, n, k, nb, d_info, linv, sA, sL, row0);
    // rows > k + nb - 1 + bw of columns k .. k + nb - 1 are zero
    const int rest = std::min(n, k + nb + bw) - (k + nb);
    if (rest > 0) {
      launch_pdl(k_trsm_panel, dim3((rest + 63) / 64, batch), 256, 0, st, A, n, k, nb, (const double*)linv, sA, sL);
      const int tiles = (rest + TB - 1) / TB;
      launch_pdl(k_syrk_update, dim3(tiles, tiles, batch), 256, 0, st, A, n, k, nb, sA);
    }
  }
  // Y = L^{-1} into work: diagonal blocks from the factorization, then the
  // off-diagonal blocks level by level (T in the scratch after linv_all)
  launch_k(k_y_init, dim3(std::max(1, 148 * 4 / batch), batch), 256, 0, st, work, n, (const double*)linv_all, sY, sL);
  double* tbuf = linv_all + sL * batch;
  for (int g = 1; g < nbk; g *= 2) {
    GemmBatch b1{}, b2{};
    b1.alpha = 1.0; b1.b_lower = 1;     // T = L21 Y11
    b1.a_bw = bw;
    b2.alpha = -1.0; b2.a_lower = 1;    // Y21 = -Y22 T
    int max_tiles = 0;
    size_t toff = 0;
    auto flush = [&]() {
      if (b1.count == 0) return;
      launch_pdl(k_gemm_batched, dim3(max_tiles, b1.count), 256, 0, st, b1);
      launch_pdl(k_gemm_batched, dim3(max_tiles, b2.count), 256, 0, st, b2);
      b1.count = b2.count = 0;
      max_tiles = 0;
    };
    for (int q = 0; q < batch; ++q) {
      double *Aq = A + sA * q, *Yq = work + sY * q;
      for (int p0 = 0; p0 < nbk; p0 += 2 * g) {
        const int r0 = p0 * NB, r1 = std::min((p0 + g) * NB, n), r2 = std::min((p0 + 2 * g) * NB, n);
        if (r1 >= r2) continue;
        const int m = r2 - r1, h = r1 - r0;
        double* T = tbuf + toff;   // distinct per pair within a level (sum of m h <= n^2 / 4 per matrix)
        toff += (size_t)m * h;
        // L21 = L[r1:r2, r0:r1] is zero below its row bw (the band), and so
        // is T: only its first mb rows are formed, and only they enter Y21
        const int mb = std::min(m, bw);
        b1.job[b1.count++] = GemmJob{Aq + (size_t)r1 * n + r0, Yq + (size_t)r0 * n + r0, T, n, n, h, mb, h, h};
        b2.job[b2.count++] = GemmJob{Yq + (size_t)r1 * n + r1, T, Yq + (size_t)r1 * n + r0, n, h, n, m, h, mb};
        max_tiles = std::max(max_tiles, ((m + TB - 1) / TB) * ((h + TB - 1) / TB));
        if (b1.count == kMaxJobs) flush();
      }
    }
    flush();
  }
  // A <- Y^T Y (lower-triangle tiles, mirrored)
  const int tiles = (n + TB - 1) / TB;
  launch_pdl(k_yty, dim3(tiles * (tiles + 1) / 2, batch), 256, 0, st, (const double*)work, A, n, sY, sA);
}

// ---------------------------------------------------------------------------
// The dissected coarsest solve.
//
// The explicit inverse of n DOFs costs n / 32 dependent block steps and n^3
// products to build and reads n^2 values at each use: on a coarsest level of
// 10,920 DOFs (25x13x9 voxels) 52 ms of a job's set-up and 368 us (FP64) a
// V-cycle.  Planes of nodes along the grid's longest axis split it instead into
// `parts` interiors and, between them, separators as thick as the stencil's
// reach, which nothing couples across.  With Z_i = A_ii^-1, C_i the coupling of
// interior i to its two separators, W_i = Z_i C_i and the Schur complement
// S = A_ss - sum C_i^T W_i,
//     x_s = S^-1 (b_s - sum W_i^T b_i),   x_i = Z_i b_i - W_i x_s,
// three products with explicit blocks: [Z_i; W_i^T] b_i, S^-1 and W_i x_s.  The
// interiors are factored as one batch, so the chain of block steps is
// (ni + ns) / 32.  Same solution, same FP64 (the FP32 V-cycle reads FP32 copies
// of the blocks and accumulates in FP64, as it does with the explicit inverse).
//   storage of part i: (ni + 2 Rm) x ni values, Z_i above W_i^T (left separator's
//   rows, then the right one's), ni padded with identity rows to the longest
//   part and a multiple of 4; then S^-1, ns x ns.
// ---------------------------------------------------------------------------
namespace {

constexpr int kMaxParts = 12;

__host__ __device__ __forceinline__ int part_planes(const DensePlan& P, int i) {
  const int T = P.planes - (P.parts - 1) * P.reach;
  return (int)((long long)(i + 1) * T / P.parts) - (int)((long long)i * T / P.parts);
}
__host__ __device__ __forceinline__ int part_first(const DensePlan& P, int i) {
  const int T = P.planes - (P.parts - 1) * P.reach;
  return (int)((long long)i * T / P.parts) + i * P.reach;
}
struct DisLoc { int part, sep, row; };   // part or sep -1; row: DOF of the node's component 0 in it
__device__ __forceinline__ DisLoc dis_locate(const DensePlan& P, int x, int y, int z) {
  const int k = P.axis == 0 ? x : (P.axis == 1 ? y : z);
  const int e = P.axis == 0 ? y + P.ny1 * z : (P.axis == 1 ? x + P.nx1 * z : x + P.nx1 * y);
  DisLoc l{-1, -1, 0};
  for (int i = 0; i < P.parts; ++i) {
    const int f = part_first(P, i), c = part_planes(P, i);
    if (k < f + c) {
      l.part = i;
      l.row = (k - f) * P.m + 3 * e;
      return l;
    }
    if (k < f + c + P.reach) {
      l.sep = i;
      l.row = i * P.rm + (k - f - c) * P.m + 3 * e;
      return l;
    }
  }
  return l;
}

// Offsets in the FP64 store and the set-up's work buffer.
__host__ __device__ __forceinline__ size_t dis_part(const DensePlan& P) { return (size_t)(P.ni + 2 * P.rm) * P.ni; }

// A_ii, C (interior x separator) and C^T, A_ss from the level's full stencil
// (27 or 125 blocks), identity on DOFs that are not free.
__global__ void k_dis_assemble(Grid c, DensePlan P, const double* __restrict__ st, const uint8_t* __restrict__ cm,
                               double* __restrict__ store, double* __restrict__ coup) {
  const int R = P.reach, W = 2 * R + 1, NBK = W * W * W, SC = NBK / 2;
  const long long nint = (long long)P.nx1 * P.ny1 * (c.lz + 1), ns = c.n;
  const size_t blk = (size_t)P.rm * P.rm;
  double* S = store + P.parts * dis_part(P);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nint * NBK;
       t += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(t / NBK), s = (int)(t % NBK);
    const int x = r % P.nx1, y = r / P.nx1 % P.ny1, z = r / (P.nx1 * P.ny1);
    const int X = x + s % W - R, Y = y + (s / W) % W - R, Z = z + s / (W * W) - R;
    if (X < 0 || X > c.lx || Y < 0 || Y > c.ly || Z < 0 || Z > c.lz) continue;
    const DisLoc a = dis_locate(P, x, y, z), b = dis_locate(P, X, Y, Z);
    const int p = c.idx(x, y, z);
    const uint8_t m = cm[p];
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) {
        double v = st[((long long)s * 9 + 3 * i + j) * ns + p];
        if (s == SC && i == j && !((m >> i) & 1)) v = 1.0;
        const int ra = a.row + i, rb = b.row + j;
        if (a.part >= 0 && b.part >= 0) {
          store[a.part * dis_part(P) + (size_t)ra * P.ni + rb] = v;
        } else if (a.sep >= 0 && b.sep >= 0) {
          S[(size_t)ra * P.ns + rb] = v;
        } else {
          // coup: per part C_left, C_left^T, C_right, C_right^T (Rm x Rm each)
          const bool in_a = a.part >= 0;
          const int part = in_a ? a.part : b.part, sep = in_a ? b.sep : a.sep;
          const int right = sep == part ? 1 : 0;   // separator i lies right of part i
          const int shift = right ? part_planes(P, part) * P.m - P.rm : 0;
          const int ii = (in_a ? ra : rb) - shift, ss = (in_a ? rb : ra) - sep * P.rm;
          double* C = coup + ((size_t)part * 4 + 2 * right) * blk;
          if (in_a) C[(size_t)ii * P.rm + ss] = v;
          else C[blk + (size_t)ss * P.rm + ii] = v;
        }
      }
  }
}
__global__ void k_dis_pad(DensePlan P, double* __restrict__ store) {
  const int i = blockIdx.y;
  for (int r = part_planes(P, i) * P.m + blockIdx.x * blockDim.x + threadIdx.x; r < P.ni; r += gridDim.x * blockDim.x)
    store[i * dis_part(P) + (size_t)r * P.ni + r] = 1.0;
}
// perm[i * ni + r]: padded-vector index of row r of part i (-1: padding); then the separators' rows
__global__ void k_dis_perm(Grid c, DensePlan P, int* __restrict__ perm) {
  const int nint = P.nx1 * P.ny1 * (c.lz + 1);
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nint; r += gridDim.x * blockDim.x) {
    const int x = r % P.nx1, y = r / P.nx1 % P.ny1, z = r / (P.nx1 * P.ny1);
    const DisLoc a = dis_locate(P, x, y, z);
    const int base = a.part >= 0 ? a.part * P.ni : P.parts * P.ni;
    for (int k = 0; k < 3; ++k) perm[base + a.row + k] = 3 * c.idx(x, y, z) + k;
  }
}

// 16 bytes of a row against the staged vector, FP64 sums
__device__ __forceinline__ double dot16(const double* row, const double* b) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(row));
  return v.x * b[0] + v.y * b[1];
}
__device__ __forceinline__ double dot16(const float* row, const double* b) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(row));
  return ((double)v.x * b[0] + (double)v.y * b[1]) + ((double)v.z * b[2] + (double)v.w * b[3]);
}
// A warp's product of a 16-byte aligned row of `n` values (a multiple of VW)
// with b in shared memory; eight loads in flight per lane.
template <typename S>
__device__ __forceinline__ double warp_row(const S* row, int n, const double* b, int lane) {
  constexpr int VW = 16 / (int)sizeof(S);
  double part[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  int j = lane * VW;
  for (; j + 7 * 32 * VW < n; j += 8 * 32 * VW) {
#pragma unroll
    for (int k = 0; k < 8; ++k) part[k] += dot16(row + j + 32 * VW * k, b + j + 32 * VW * k);
  }
  for (; j < n; j += 32 * VW) part[7] += dot16(row + j, b + j);
  double s = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

constexpr int kDisRows = 32;   // rows per block: the staged vector serves four rows a warp

// y_i = [Z_i; W_i^T] b_i
template <typename T, typename S>
__global__ void __launch_bounds__(256) k_dis_parts(DensePlan P, const S* __restrict__ store,
                                                   const int* __restrict__ perm, const T* b,
                                                   double* __restrict__ y, const KrylovState* ks) {
  pdl_enter();
  if (ks && ks->done) return;
  extern __shared__ double sb[];
  const int i = blockIdx.y, rows = P.ni + 2 * P.rm;
  for (int k = threadIdx.x; k < P.ni; k += blockDim.x) {
    const int q = __ldg(perm + i * P.ni + k);
    sb[k] = q >= 0 ? (double)b[q] : 0.0;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const S* M = store + i * dis_part(P);
  for (int r = blockIdx.x * kDisRows + warp; r < min(rows, (int)(blockIdx.x + 1) * kDisRows); r += 8) {
    const double v = warp_row<S>(M + (size_t)r * P.ni, P.ni, sb, lane);
    if (lane == 0) y[(size_t)i * rows + r] = v;
  }
}
// x_s = S^-1 (b_s - the parts' W^T b); S in rows of ld values
template <typename T, typename S>
__global__ void __launch_bounds__(256) k_dis_schur(DensePlan P, const S* __restrict__ Sinv, int ld,
                                                   const int* __restrict__ perm, const T* b, const double* y,
                                                   double* __restrict__ xs,
                                                   T* __restrict__ x, const KrylovState* ks) {
  pdl_enter();
  if (ks && ks->done) return;
  extern __shared__ double sb[];
  const int rows = P.ni + 2 * P.rm;
  for (int k = threadIdx.x; k < ld; k += blockDim.x) {
    double v = 0.0;
    if (k < P.ns) {
      const int sep = k / P.rm, l = k - sep * P.rm;
      v = (double)b[__ldg(perm + P.parts * P.ni + k)] - y[(size_t)sep * rows + P.ni + P.rm + l] -
          y[(size_t)(sep + 1) * rows + P.ni + l];
    }
    sb[k] = v;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = blockIdx.x * 8 + warp; r < P.ns; r += gridDim.x * 8) {
    const double v = warp_row<S>(Sinv + (size_t)r * ld, ld, sb, lane);
    if (lane == 0) {
      xs[r] = v;
      x[__ldg(perm + P.parts * P.ni + r)] = (T)v;
    }
  }
}
// x_i = (Z_i b_i) - W_i x_s: lanes take 32 rows, warps share the separators' DOFs
template <typename T, typename S>
__global__ void __launch_bounds__(256) k_dis_back(DensePlan P, const S* __restrict__ store,
                                                  const int* __restrict__ perm, const double* y, const double* xs,
                                                  T* __restrict__ x,
                                                  const KrylovState* ks) {
  pdl_enter();
  if (ks && ks->done) return;
  __shared__ double part[8][33];
  const int i = blockIdx.y, rows = P.ni + 2 * P.rm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = blockIdx.x * 32 + lane;
  const S* W = store + i * dis_part(P) + (size_t)P.ni * P.ni;
  const int c0 = i > 0 ? 0 : P.rm, c1 = i + 1 < P.parts ? 2 * P.rm : P.rm;
  const double* xl = xs + (long long)(i - 1) * P.rm;   // column c belongs to row c of the pair (separators i - 1, i)
  double s = 0.0;
  if (r < P.ni) {
#pragma unroll 8
    for (int c = c0 + warp; c < c1; c += 8) s += (double)__ldg(W + (size_t)c * P.ni + r) * xl[c];
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && r < P.ni) {
    const int q = __ldg(perm + i * P.ni + r);
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w][lane];
    if (q >= 0) x[q] = (T)(y[(size_t)i * rows + r] - t);
  }
}

}  // namespace

// The cheapest split by a model of the set-up and 80 uses, in microseconds:
// 60 per block step of 32 columns, 2.5e-8 per n^3 (both measured on 10,920
// DOFs: 342 steps, 32 ms of products), 8 bytes per value read at 4.5 TB/s, and
// for a split 150 of set-up launches and 8 per use for the two more kernels.
// It splits 10,920 DOFs into 7 parts of 1,260 (a 100x52x36 job, FP64: 99 -> 34 ms).
// Whole set-up and 80 V-cycles of FP64 two-level solvers, as chosen / explicit
// inverse, ms: 735 DOFs one piece 4.35, 945 4.80 / 4.71, 1,155 4.65 / 5.14, 2,835 6.7 /
// 8.4, 4,563 9.0 / 15.6, 9,405 16.9 / 54.6, 15,249 31 / 216; reach 2: 1,617 10.6 / 10.5, 3,159
// 13.9 / 16.8, 14,625 57 / 230.  No other number of parts was more than 2 % better.
DensePlan dense_plan(const Grid& c, int reach) {
  DensePlan best{};
  const int dims[3] = {c.lx + 1, c.ly + 1, c.lz + 1};
  best.n = 3 * dims[0] * dims[1] * dims[2];
  best.parts = 1;
  best.ni = best.n;
  const double n = best.n;
  double least = n / 32 * 60 + n * n * n * 2.5e-8 + 80 * (n * n * 8 / 4.5e6);
  int axis = 0;
  for (int a = 1; a < 3; ++a)
    if (dims[a] > dims[axis]) axis = a;
  for (int parts = 2; parts <= kMaxParts; ++parts) {
    DensePlan P{};
    P.n = best.n;
    P.axis = axis;
    P.reach = reach < 1 ? 1 : reach;
    P.parts = parts;
    P.planes = dims[axis];
    P.nx1 = dims[0];
    P.ny1 = dims[1];
    P.m = P.n / dims[axis];
    P.rm = P.reach * P.m;
    const int inner = P.planes - (parts - 1) * P.reach;
    if (inner < parts * P.reach) break;   // a part at least as thick as the reach keeps its separators apart
    P.ni = ((inner + parts - 1) / parts * P.m + 3) / 4 * 4;
    P.ns = (parts - 1) * P.rm;
    if (P.ns % 2) continue;   // rows of S^-1 start on 16 bytes
    const double ni = P.ni, ns = P.ns, rm = P.rm;
    const double cost = 150 + (ni + ns) / 32 * 60 + (parts * ni * ni * ni + ns * ns * ns) * 2.5e-8 +
                        80 * (8 + (parts * (ni * ni + 4 * rm * ni) + ns * ns) * 8 / 4.5e6);
    if (cost < least) {
      least = cost;
      best = P;
    }
  }
  return best;
}

size_t dense_store_count(const DensePlan& P) {
  return P.parts == 1 ? (size_t)P.n * P.n : P.parts * dis_part(P) + (size_t)P.ns * P.ns;
}
size_t dense_store32_count(const DensePlan& P) {
  return P.parts == 1 ? (size_t)P.n * dense_ld32(P.n) : P.parts * dis_part(P) + (size_t)P.ns * dense_ld32(P.ns);
}
size_t dense_perm_count(const DensePlan& P) { return P.parts == 1 ? (size_t)P.n : (size_t)P.parts * P.ni + P.ns; }
size_t dense_vec_count(const DensePlan& P) {
  return P.parts == 1 ? 1 : (size_t)P.parts * (P.ni + 2 * P.rm) + P.ns;
}
size_t dense_work_count(const DensePlan& P) {
  if (P.parts == 1) return cholesky_work(P.n, 1);
  return std::max(cholesky_work(P.ni, P.parts), cholesky_work(P.ns, 1)) + (size_t)P.parts * 4 * P.rm * P.rm;
}
void launch_dense_perm(const Grid& c, const DensePlan& P, int* perm, cudaStream_t st) {
  if (P.parts == 1) {
    launch_k(k_dense_perm, (P.n + 255) / 256, 256, 0, st, c, perm, P.n);
    return;
  }
  cudaMemsetAsync(perm, 0xff, sizeof(int) * dense_perm_count(P), st);
  launch_k(k_dis_perm, (P.n / 3 + 255) / 256, 256, 0, st, c, P, perm);
}

// The coarsest operator's explicit inverse, or the dissected one's blocks, in
// `store`, from the level's full stencil.  d_info: kDenseNoRow, or the index in
// the permutation table of the first row without a positive pivot.
void dense_build(const Grid& c, const DensePlan& P, const double* stencil, int reach, const uint8_t* cmask,
                 double* store, double* work, int* d_info, cudaStream_t st) {
  cudaMemsetAsync(d_info, 0x7f, sizeof(int), st);   // (kDenseNoRow)
  if (P.parts == 1) {
    if (reach > 1) wide_dense_assemble(c, reach, stencil, cmask, store, P.n, st);
    else dense_assemble(c, stencil, cmask, store, P.n, st);
    // DOF bandwidth of the reach-R stencil in reference node order
    const long long nx1 = c.lx + 1, ny1 = c.ly + 1;
    const long long bw = 3LL * std::max(reach, 1) * (1 + nx1 + nx1 * ny1) + 2;
    cholesky_inverse(store, work, P.n, (int)std::min<long long>(bw, P.n), d_info, st, 1, 0, 0);
    return;
  }
  const size_t sp = dis_part(P), blk = (size_t)P.rm * P.rm;
  double* coup = work + std::max(cholesky_work(P.ni, P.parts), cholesky_work(P.ns, 1));
  double* S = store + P.parts * sp;
  cudaMemsetAsync(store, 0, sizeof(double) * dense_store_count(P), st);
  cudaMemsetAsync(coup, 0, sizeof(double) * P.parts * 4 * blk, st);
  const int W = 2 * P.reach + 1;
  const long long pairs = (long long)(P.n / 3) * W * W * W;
  launch_k(k_dis_assemble, (int)std::min<long long>((pairs + 255) / 256, 148LL * 64), 256, 0, st, c, P, stencil, cmask,
           store, coup);
  launch_k(k_dis_pad, dim3(4, P.parts), 256, 0, st, P, store);
  // within a part the DOFs run plane by plane: the band is reach + 1 planes
  cholesky_inverse(store, work, P.ni, P.rm + P.m, d_info, st, P.parts, sp, 0);
  GemmBatch w{}, r{}, l{};
  w.alpha = 1.0;
  r.alpha = l.alpha = -1.0;
  r.beta = l.beta = 1.0;
  const int rm = P.rm, ni = P.ni;
  for (int i = 0; i < P.parts; ++i) {
    double *Z = store + i * sp, *WL = Z + (size_t)ni * ni, *WR = WL + (size_t)rm * ni, *C = coup + (size_t)i * 4 * blk;
    const int last = part_planes(P, i) * P.m - rm;   // first row of the planes next to the right separator
    // W^T = C^T Z (Z is symmetric); S -= W^T C, the lower blocks
    if (i > 0) w.job[w.count++] = GemmJob{C + blk, Z, WL, rm, ni, ni, rm, ni, rm};
    if (i + 1 < P.parts) w.job[w.count++] = GemmJob{C + 3 * blk, Z + (size_t)last * ni, WR, rm, ni, ni, rm, ni, rm};
    double* Sii = S + (size_t)i * rm * P.ns + (size_t)i * rm;   // separator i against itself
    if (i + 1 < P.parts) r.job[r.count++] = GemmJob{WR + last, C + 2 * blk, Sii, ni, rm, P.ns, rm, rm, rm};
    if (i > 0) {
      l.job[l.count++] = GemmJob{WL, C, Sii - (size_t)rm * P.ns - rm, ni, rm, P.ns, rm, rm, rm};
      if (i + 1 < P.parts) l.job[l.count++] = GemmJob{WR, C, Sii - rm, ni, rm, P.ns, rm, rm, rm};
    }
  }
  const int t = (rm + TB - 1) / TB;
  launch_pdl(k_gemm_batched, dim3(t * ((ni + TB - 1) / TB), w.count), 256, 0, st, w);
  launch_pdl(k_gemm_batched, dim3(t * t, r.count), 256, 0, st, r);
  launch_pdl(k_gemm_batched, dim3(t * t, l.count), 256, 0, st, l);
  cholesky_inverse(S, work, P.ns, 2 * rm, d_info, st, 1, 0, P.parts * P.ni);
}
void dense_build32(const DensePlan& P, const double* store, float* store32, cudaStream_t st) {
  const size_t head = P.parts == 1 ? 0 : P.parts * dis_part(P);
  const int n = P.parts == 1 ? P.n : P.ns;
  if (head) launch_convert<double, float>(store, store32, (long long)head, st);
  const long long total = (long long)n * dense_ld32(n);
  launch_k(k_convert_pad, (int)std::min<long long>((total + 255) / 256, 148LL * 32), 256, 0, st, store + head,
           store32 + head, n, dense_ld32(n));
}

template <typename T, typename S>
static void dissected_solve(const DensePlan& P, const S* store, int ld, const int* perm, double* vec, const T* b, T* x,
                            const KrylovState* ks, cudaStream_t st) {
  double* xs = vec + (size_t)P.parts * (P.ni + 2 * P.rm);
  launch_pdl(k_dis_parts<T, S>, dim3((P.ni + 2 * P.rm + kDisRows - 1) / kDisRows, P.parts), 256, sizeof(double) * P.ni, st,
           P, store, perm, b, vec, ks);
  launch_pdl(k_dis_schur<T, S>, (P.ns + 7) / 8, 256, sizeof(double) * ld, st, P, store + P.parts * dis_part(P), ld, perm, b,
           (const double*)vec, xs, x, ks);
  launch_pdl(k_dis_back<T, S>, dim3((P.ni + 31) / 32, P.parts), 256, 0, st, P, store, perm, (const double*)vec,
           (const double*)xs, x, ks);
}

// b is staged in dynamic shared memory (n doubles, n <= 16384).  The limit is
// a per-function attribute shared by every solver of the process (solvers of
// different sizes run concurrently in batch solves): always the maximum.
void dense_prepare_smem() {
  const int bytes = (int)sizeof(double) * 16384;
  auto allow = [&](const void* f) { cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
  allow((const void*)k_dense_solve);
  allow((const void*)k_dense_solve_f32);
  allow((const void*)k_dis_parts<double, double>);
  allow((const void*)k_dis_parts<float, float>);
  allow((const void*)k_dis_schur<double, double>);
  allow((const void*)k_dis_schur<float, float>);
}

int dense_ld32(int n) { return (n + 3) / 4 * 4; }

template <>
void launch_dense_solve<double>(const DensePlan& P, const double* store, const float*, const int* perm, double* vec,
                                const double* b, double* x, const KrylovState* ks, cudaStream_t st) {
  if (P.parts > 1) {
    // (ns is even or its rows would not start on 16 bytes: see dense_plan)
    dissected_solve<double, double>(P, store, P.ns, perm, vec, b, x, ks, st);
    return;
  }
  launch_pdl(k_dense_solve, (P.n + 7) / 8, 256, sizeof(double) * P.n, st, store, P.n, perm, b, x, ks);
}
template <>
void launch_dense_solve<float>(const DensePlan& P, const double*, const float* store32, const int* perm, double* vec,
                               const float* b, float* x, const KrylovState* ks, cudaStream_t st) {
  if (P.parts > 1) {
    dissected_solve<float, float>(P, store32, dense_ld32(P.ns), perm, vec, b, x, ks, st);
    return;
  }
  const int ld = dense_ld32(P.n);
  launch_pdl(k_dense_solve_f32, (P.n + 7) / 8, 256, sizeof(double) * ld, st, store32, P.n, ld, perm, b, x, ks);
}

}  // namespace vf
