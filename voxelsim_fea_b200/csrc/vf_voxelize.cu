// Point-in-mesh inside test (voxelization), the step before grid assembly
// (the reference's core/inside_worker.py:_inside_mask_numpy, lines 105-147).
//
// One fixed ray direction d per query; a point is inside a closed triangle
// mesh when the ray from it crosses an odd number of triangles
// (Moeller-Trumbore: u >= -1e-7, v >= -1e-7, u + v <= 1 + 1e-7, t > 1e-7,
// triangles with |det| < 1e-9 skipped).  Triangles are pre-transformed once
// (v0, e1, e2, p = d x e2, 1/det).  Every product and sum is an explicitly rounded FP64
// operation in the reference's evaluation order (no contraction into FMAs),
// so the inside/outside decisions are the reference's bit for bit.
//
// Given points: one thread per point, every triangle streamed through shared
// memory (k_inside).  Points of a voxel grid (voxel centers in element order
// iz-fastest, or nodes in node order x-fastest: inside_worker.py:voxel_centers /
// node_coords): each triangle visits only the grid points whose ray can meet
// it (k_inside_grid), found from the bounds of its projection along the ray,
// widened by the test's own tolerance and a bound of its rounding, and flips
// their parity; the test of a visited point is the same arithmetic, and a
// point that is not visited could not have passed it.  All points against all
// triangles cost points x triangles tests at the FP64 rate (786,432 centers x
// 10,000 triangles: 18.8 ms); now their number is the grid lines that each
// triangle covers times the points before it.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "../../include/voxfea.h"
#include "vf_common.cuh"
#include "vf_workspace.cuh"

namespace vf {

namespace {

constexpr int kTile = 128;   // triangles per shared-memory tile
constexpr int kTriVals = 13; // v0 (3), e1 (3), e2 (3), pvec (3), inv_det (1)

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
// a.b = (a0 b0 + a1 b1) + a2 b2
__device__ __forceinline__ double dot3(const double* a, const double* b) {
  return add(add(mul(a[0], b[0]), mul(a[1], b[1])), mul(a[2], b[2]));
}
// a x b, component-wise a1 b2 - a2 b1, ...
__device__ __forceinline__ void cross3(const double* a, const double* b, double* c) {
  c[0] = sub(mul(a[1], b[2]), mul(a[2], b[1]));
  c[1] = sub(mul(a[2], b[0]), mul(a[0], b[2]));
  c[2] = sub(mul(a[0], b[1]), mul(a[1], b[0]));
}

struct Dir { double d[3]; };

// Whether the ray from p meets prepared triangle T (T[12] != 0).
__device__ __forceinline__ bool hits_triangle(const double* p, const double* T, const Dir& dir) {
  const double inv = T[12];
  const double tv[3] = {sub(p[0], T[0]), sub(p[1], T[1]), sub(p[2], T[2])};
  const double u = mul(dot3(tv, T + 9), inv);
  double q[3];
  cross3(tv, T + 3, q);
  const double v = mul(dot3(dir.d, q), inv);
  const double t = mul(dot3(T + 6, q), inv);
  return u >= -1e-7 && v >= -1e-7 && add(u, v) <= 1.0 + 1e-7 && t > 1e-7;
}

// Coordinate c of grid point k along its axis (mode 1: centers, 2: nodes).
__device__ __forceinline__ double grid_coord(int mode, int k, double vs, double o) {
  return add(mul(mode == 1 ? k + 0.5 : (double)k, vs), o);
}

__global__ void k_prepare_tris(const double* __restrict__ verts, const int64_t* __restrict__ faces, int64_t nf,
                               Dir dir, double* __restrict__ tri) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nf; t += (int64_t)gridDim.x * blockDim.x) {
    double v0[3], v1[3], v2[3], e1[3], e2[3], pv[3];
    for (int c = 0; c < 3; ++c) {
      v0[c] = verts[3 * faces[3 * t] + c];
      v1[c] = verts[3 * faces[3 * t + 1] + c];
      v2[c] = verts[3 * faces[3 * t + 2] + c];
      e1[c] = sub(v1[c], v0[c]);
      e2[c] = sub(v2[c], v0[c]);
    }
    cross3(dir.d, e2, pv);
    const double det = dot3(e1, pv);
    const bool parallel = fabs(det) < 1e-9;
    double* o = tri + kTriVals * t;
    for (int c = 0; c < 3; ++c) { o[c] = v0[c]; o[3 + c] = e1[c]; o[6 + c] = e2[c]; o[9 + c] = pv[c]; }
    o[12] = parallel ? 0.0 : 1.0 / det;   // 0 marks a skipped triangle
  }
}

// mode 0: explicit points (x, y, z) triples; 1: voxel centers; 2: grid nodes
__global__ void k_inside(int mode, const double* __restrict__ pts, int64_t npts, int nx, int ny, int nz,
                         double ox, double oy, double oz, double vs, const double* __restrict__ tri, int64_t nf,
                         Dir dir, uint8_t* __restrict__ out) {
  __shared__ double s_tri[kTile * kTriVals];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double p[3] = {0.0, 0.0, 0.0};
  const bool live = i < npts;
  if (live) {
    if (mode == 0) {
      p[0] = pts[3 * i]; p[1] = pts[3 * i + 1]; p[2] = pts[3 * i + 2];
    } else {   // element order (ix * ny + iy) * nz + iz, node order ix + (nx+1) (iy + (ny+1) iz)
      const int nxp = nx + 1, nyp = ny + 1;
      const int ix = mode == 1 ? (int)(i / ((int64_t)nz * ny)) : (int)(i % nxp);
      const int iy = mode == 1 ? (int)((i / nz) % ny) : (int)((i / nxp) % nyp);
      const int iz = mode == 1 ? (int)(i % nz) : (int)(i / ((int64_t)nxp * nyp));
      p[0] = grid_coord(mode, ix, vs, ox);
      p[1] = grid_coord(mode, iy, vs, oy);
      p[2] = grid_coord(mode, iz, vs, oz);
    }
  }
  int hits = 0;
  for (int64_t t0 = 0; t0 < nf; t0 += kTile) {
    const int nt = (int)((nf - t0 < kTile) ? (nf - t0) : kTile);
    __syncthreads();
    for (int k = threadIdx.x; k < nt * kTriVals; k += blockDim.x) s_tri[k] = tri[kTriVals * t0 + k];
    __syncthreads();
    if (!live) continue;
    for (int k = 0; k < nt; ++k) {
      const double* T = s_tri + kTriVals * k;
      if (T[12] == 0.0) continue;   // |det| < 1e-9
      hits += hits_triangle(p, T, dir) ? 1 : 0;
    }
  }
  if (live) out[i] = (uint8_t)(hits & 1);
}

// The grid of k_inside_grid: n points along each axis, the ray's dominant axis
// a and the other two b, c; sb, sc: the ray's slopes along them.
struct RayGrid {
  int mode, n[3], a, b, c;
  double o[3], vs, sb, sc;
};

// The points that one triangle's test can pass, as ranges of the projected
// coordinates B = p_b - sb p_a and C = p_c - sc p_a (constant along the ray)
// and of p_a.  A point passes only if, in exact arithmetic,
//   p + t d = v0 + u e1 + v e2,  u, v >= -tau, u + v <= 1 + tau, t >= -tau_t
// with tau the test's 1e-7 plus what rounding can add: u and v are sums of a
// few products of |tv| <= R, |e1|, |e2|, |d| times 1/det, each within 16 eps
// of them and 1/det itself within 16 eps |e1| |e2| |d| / |det| of its own
// (64 eps here).  So B lies within 3 tau (|B(e1)| + |B(e2)|) of the vertices'
// range.  Bounds that are not finite come out as the whole axis.
struct TriBounds { double b0, b1, c0, c1, amin, amax; };
__device__ __forceinline__ TriBounds tri_bounds(const double* T, const Dir& dir, const RayGrid& G) {
  auto norm1 = [](const double* v) { return fabs(v[0]) + fabs(v[1]) + fabs(v[2]); };
  double R = 0.0;
  for (int k = 0; k < 3; ++k) {
    const double lo = G.o[k], hi = G.o[k] + G.n[k] * G.vs;
    R += fmax(fabs(lo - T[k]), fabs(hi - T[k])) + fabs(lo) * 1e-15 + fabs(T[k]) * 1e-15;
  }
  const double l1 = norm1(T + 3), l2 = norm1(T + 6), ld = norm1(dir.d);
  const double eps = 64.0 * 2.3e-16 * fabs(T[12]) * ld;
  const double S = R + l1 + l2;
  const double tau = 4e-7 + eps * S * (l1 + l2), tau_t = eps / ld * S * l1 * l2 + 1e-7;
  auto B = [&](const double* v) { return v[G.b] - G.sb * v[G.a]; };
  auto C = [&](const double* v) { return v[G.c] - G.sc * v[G.a]; };
  const double vb = B(T), vc = C(T), b1 = B(T + 3), b2 = B(T + 6), c1 = C(T + 3), c2 = C(T + 6);
  // (the projections' own rounding, and 1e-6 of a voxel for the index arithmetic)
  const double slack = 1e-6 * G.vs + 1e-14 * (norm1(T) + R);
  const double mb = 3.0 * tau * (fabs(b1) + fabs(b2)) + slack, mc = 3.0 * tau * (fabs(c1) + fabs(c2)) + slack;
  const double a1 = T[3 + G.a], a2 = T[6 + G.a];
  const double ma = 3.0 * tau * (fabs(a1) + fabs(a2)) + tau_t * fabs(dir.d[G.a]) + slack;
  TriBounds r;
  r.b0 = vb + fmin(0.0, fmin(b1, b2)) - mb;
  r.b1 = vb + fmax(0.0, fmax(b1, b2)) + mb;
  r.c0 = vc + fmin(0.0, fmin(c1, c2)) - mc;
  r.c1 = vc + fmax(0.0, fmax(c1, c2)) + mc;
  r.amin = T[G.a] + fmin(0.0, fmin(a1, a2)) - ma;
  r.amax = T[G.a] + fmax(0.0, fmax(a1, a2)) + ma;
  return r;
}
// first / last grid index whose coordinate is >= lo / <= hi (NaN: the whole axis)
__device__ __forceinline__ int first_index(double lo, double o, double vs, double half, int n) {
  return (int)fmin(fmax(ceil((lo - o) / vs - half), 0.0), (double)n);
}
__device__ __forceinline__ int last_index(double hi, double o, double vs, double half, int n) {
  return (int)fmax(fmin(floor((hi - o) / vs - half), (double)(n - 1)), -1.0);
}

// blockIdx.x: triangle; the blocks of a triangle (gridDim.y) share its
// candidate points: the grid positions along the ray's axis times the widest
// rectangle of grid lines its projection covers at any of them.
__global__ void __launch_bounds__(128) k_inside_grid(RayGrid G, const double* __restrict__ tri, Dir dir,
                                                     unsigned* __restrict__ out) {
  const double* Tg = tri + (int64_t)kTriVals * blockIdx.x;
  double T[kTriVals];
#pragma unroll
  for (int k = 0; k < kTriVals; ++k) T[k] = __ldg(Tg + k);
  if (T[12] == 0.0) return;
  const TriBounds r = tri_bounds(T, dir, G);
  const double half = G.mode == 1 ? 0.5 : 0.0;
  const int na = G.n[G.a], nb = G.n[G.b], nc = G.n[G.c];
  // the ray runs along +a or -a: points before the triangle's far end
  int ia0 = 0, ia1 = na - 1;
  if (dir.d[G.a] > 0.0) ia1 = last_index(r.amax, G.o[G.a], G.vs, half, na);
  else ia0 = first_index(r.amin, G.o[G.a], G.vs, half, na);
  const int la = ia1 - ia0 + 1;
  if (la <= 0) return;
  const int wb = (int)fmin(floor((r.b1 - r.b0) / G.vs) + 2.0, (double)nb);
  const int wc = (int)fmin(floor((r.c1 - r.c0) / G.vs) + 2.0, (double)nc);
  const int64_t total = (int64_t)la * wb * wc;
  for (int64_t i = blockIdx.y * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.y * blockDim.x) {
    int64_t q = i / wc;
    const int jc = (int)(i - q * wc), ja = (int)(q / wb), jb = (int)(q - (int64_t)ja * wb);
    int k[3];
    double p[3];
    k[G.a] = ia0 + ja;
    p[G.a] = grid_coord(G.mode, k[G.a], G.vs, G.o[G.a]);
    const double sb = G.sb * p[G.a], sc = G.sc * p[G.a];
    k[G.b] = first_index(r.b0 + sb, G.o[G.b], G.vs, half, nb) + jb;
    k[G.c] = first_index(r.c0 + sc, G.o[G.c], G.vs, half, nc) + jc;
    if (k[G.b] >= nb || k[G.c] >= nc) continue;
    p[G.b] = grid_coord(G.mode, k[G.b], G.vs, G.o[G.b]);
    p[G.c] = grid_coord(G.mode, k[G.c], G.vs, G.o[G.c]);
    if (!hits_triangle(p, T, dir)) continue;
    const int64_t e = G.mode == 1 ? ((int64_t)k[0] * G.n[1] + k[1]) * G.n[2] + k[2]
                                  : k[0] + (int64_t)G.n[0] * (k[1] + (int64_t)G.n[1] * k[2]);
    atomicXor(out + (e >> 2), 1u << (8 * (e & 3)));   // one byte per point
  }
}

int inside_run(int mode, const double* verts, int64_t nv, const int64_t* faces, int64_t nf, const double* pts,
               int64_t npts, const int32_t* dims, const double* origin, double vsize, const double* dir3,
               uint8_t* out) {
  if (npts <= 0) return VF_OK;
  for (int64_t k = 0; k < 3 * nf; ++k)   // the kernels index verts by these: check them here
    if (faces[k] < 0 || faces[k] >= nv) return VF_ERR_ARG;
  Workspace ws;
  if (!ws.open()) return VF_ERR_CUDA;
  cudaStream_t st = ws.st;
  double *d_v = nullptr, *d_tri = nullptr, *d_p = nullptr;
  int64_t* d_f = nullptr;
  uint8_t* d_o = nullptr;
  const size_t nfs = (size_t)(nf > 0 ? nf : 1);
  if (!ws.alloc(&d_v, 3 * (size_t)(nv > 0 ? nv : 1)) || !ws.alloc(&d_f, 3 * nfs) || !ws.alloc(&d_tri, kTriVals * nfs) ||
      !ws.alloc(&d_o, (size_t)npts) || (mode == 0 && !ws.alloc(&d_p, 3 * (size_t)npts)))
    return VF_ERR_NOMEM;
  Dir d;
  for (int c = 0; c < 3; ++c) d.d[c] = dir3[c];
  if (nf > 0) {
    cudaMemcpyAsync(d_v, verts, sizeof(double) * 3 * (size_t)nv, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_f, faces, sizeof(int64_t) * 3 * (size_t)nf, cudaMemcpyHostToDevice, st);
    launch_k(k_prepare_tris, (int)((nf + 255) / 256 < 4096 ? (nf + 255) / 256 : 4096), 256, 0, st,
             (const double*)d_v, (const int64_t*)d_f, nf, d, d_tri);
  }
  if (mode == 0) cudaMemcpyAsync(d_p, pts, sizeof(double) * 3 * (size_t)npts, cudaMemcpyHostToDevice, st);
  const int nx = dims ? dims[0] : 0, ny = dims ? dims[1] : 0, nz = dims ? dims[2] : 0;
  const double ox = origin ? origin[0] : 0.0, oy = origin ? origin[1] : 0.0, oz = origin ? origin[2] : 0.0;
  int axis = 0;
  for (int c = 1; c < 3; ++c)
    if (std::fabs(dir3[c]) > std::fabs(dir3[axis])) axis = c;
  const int64_t kMaxTri = 1 << 30;   // a block each
  if (mode == 0 || nf > kMaxTri || !(vsize > 0.0) || !(std::fabs(dir3[axis]) > 0.0) || !std::isfinite(dir3[0] + dir3[1] + dir3[2])) {
    // given points, or a grid or ray that has no lines to speak of
    launch_k(k_inside, (unsigned)((npts + 255) / 256), 256, 0, st, mode, (const double*)d_p, npts, nx, ny, nz, ox, oy,
             oz, vsize, (const double*)d_tri, nf, d, d_o);
  } else {
    cudaMemsetAsync(d_o, 0, (size_t)npts, st);
    RayGrid G;
    G.mode = mode;
    for (int c = 0; c < 3; ++c) {
      G.n[c] = dims[c] + (mode == 2 ? 1 : 0);
      G.o[c] = origin[c];
    }
    G.a = axis; G.b = (axis + 1) % 3; G.c = (axis + 2) % 3;
    G.vs = vsize;
    G.sb = dir3[G.b] / dir3[axis];
    G.sc = dir3[G.c] / dir3[axis];
    // a mesh of few triangles (a support box: 12) covers many points with each:
    // enough blocks to fill the device share a triangle's candidates
    const unsigned per = (unsigned)std::max<int64_t>(1, std::min<int64_t>((16 * 148 + nf - 1) / std::max<int64_t>(nf, 1), 256));
    if (nf > 0)
      launch_k(k_inside_grid, dim3((unsigned)nf, per), 128, 0, st, G, (const double*)d_tri, d, (unsigned*)d_o);
  }
  cudaMemcpyAsync(out, d_o, (size_t)npts, cudaMemcpyDeviceToHost, st);
  return cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess ? VF_ERR_CUDA : VF_OK;
}

}  // namespace

}  // namespace vf

extern "C" {

int vf_inside_points(const double* verts, int64_t nv, const int64_t* faces, int64_t nf, const double* points,
                     int64_t npts, const double* dir3, uint8_t* out) {
  if (npts < 0 || nf < 0 || nv < 0 || !dir3 || (npts > 0 && (!points || !out)) || (nf > 0 && (!verts || !faces)))
    return VF_ERR_ARG;
  return vf::inside_run(0, verts, nv, faces, nf, points, npts, nullptr, nullptr, 0.0, dir3, out);
}

int vf_inside_grid(const double* verts, int64_t nv, const int64_t* faces, int64_t nf, const int32_t* dims3,
                   const double* origin3, double vsize, int32_t target, const double* dir3, uint8_t* out) {
  if (!dims3 || !origin3 || !dir3 || !out || nf < 0 || nv < 0 || (nf > 0 && (!verts || !faces)) ||
      (target != 0 && target != 1) || dims3[0] < 1 || dims3[1] < 1 || dims3[2] < 1)
    return VF_ERR_ARG;
  const int64_t n = target == 0 ? (int64_t)dims3[0] * dims3[1] * dims3[2]
                                : (int64_t)(dims3[0] + 1) * (dims3[1] + 1) * (dims3[2] + 1);
  return vf::inside_run(target == 0 ? 1 : 2, verts, nv, faces, nf, nullptr, n, dims3, origin3, vsize, dir3, out);
}

}  // extern "C"
