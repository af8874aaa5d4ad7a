// Geometric multigrid preconditioner for the lattice Jacobian (sm_100a).
//
// The structured-lattice counterpart of the BoomerAMG preconditioner the reference puts
// in its Jacobian solves (algorithms/linSolvers.py:243-828): a symmetric V-cycle over
//   level 0   the Q2 lattice itself (the matrix-free operator and its Jacobi diagonal),
//   level 1   Q1 on the same elements (the Q2 lattice's vertices),
//   level l   Q1 on elements coarsened 2:1 while every axis stays even and >= 4,
// with Chebyshev-Jacobi smoothing (degree s before and after, the same polynomial, so the
// cycle is symmetric and positive: a fixed linear preconditioner for CG) and a
// Chebyshev solve of higher degree on the coarsest level.  Between any two levels the
// node lattices are 2:1 (F = 2C - 1 nodes per axis: the Q1 space is nested in Q2 and in
// the next finer Q1), so one trilinear prolongation P and its transpose R = P^T (full
// weighting) serve every pair.  Coarse operators are rediscretised: Q1 stiffness with
// one coefficient per element, the Gauss-weighted mean of e^m over the Q2 element
// (level 1), the mean of the 8 children above.  The Dirichlet nodes must be the whole
// boundary: eliminated rows are the identity on every level and restricted residuals
// are zero there.  The set-up is FP64; the cycle runs in FP64 or, on request, in FP32
// on single-precision copies of the level data (the caller's residual read and the result
// written in FP64, the CG around it unchanged).  Deterministic, and free of host
// synchronisation after set-up, so a CG iteration with its V-cycle can be captured as a
// CUDA graph.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <new>
#include <type_traits>
#include <utility>
#include <vector>

#include "hm_common.cuh"
#include "hm_internal.h"

namespace hm {

// a level in the cycle's precision T (the set-up keeps an FP64 copy of every level)
template <typename T>
struct MGLevelT {
  int nx, ny, nz;        // elements
  int Nx, Ny, Nz;        // nodes per axis
  double hx, hy, hz;     // element sizes
  int64_t nodes, elems;
  T* coef;               // per element (levels >= 1)
  T* diag;               // Jacobi diagonal (level 0: the caller's; FP64 levels only)
  T* idiag;              // its reciprocal, by which the smoothers multiply
  T *x, *b, *r, *d, *t;
  double* cheb;          // Chebyshev on the device: [0] theta (d0 = r / (theta diag)),
                         // [1 + k] c1_k, [1 + kChebMax + k] c2_k (d = c1 d + c2 r / diag)
  int degree;
  T* cinv;               // coarsest level with few interior nodes: the inverse of its
                         // interior block (row-major), solved exactly; else nullptr
};
using MGLevel = MGLevelT<double>;
constexpr int kChebMax = 40;

}  // namespace hm

struct hm_mg {
  hm::Lattice L;
  int nlev;
  hm::MGLevel lv[16];
  void* jac;             // level-0 operator data (FP64, from hm_lattice_jacobian_prepare)
  const uint8_t* ess;
  int degree, coarse_degree;
  double* scratch;       // partial sums of the set-up's inner products, their counter
  const uint8_t* checked_ess;   // the markers last found to be the whole boundary
  int tail_first;        // first level of the one-launch tail (nlev: none)
  int64_t tail_nodes;    // its levels' nodes at most
  int fused;             // smoothing steps fused with their operator pass
  // the FP32 cycle (single != 0): every level's vectors, coefficients, reciprocal
  // diagonal and coarse inverse in single precision, refreshed from the FP64 set-up; the
  // level-0 operator data (the points' D) in jac32
  int single;
  hm::MGLevelT<float> lv32[16];
  float* jac32;
};

namespace hm {

constexpr int kMGBlocks = 296;

__device__ __forceinline__ bool on_boundary(int i, int j, int k, int Nx, int Ny, int Nz) {
  return i == 0 || j == 0 || k == 0 || i == Nx - 1 || j == Ny - 1 || k == Nz - 1;
}

// a product rounded on its own (no contraction into a neighbouring add)
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// A node of a level by its number (32-bit: the lattice keeps every index below 2^31).
struct MGNode { int i, j, k; };
template <typename T>
__device__ __forceinline__ MGNode node_at(const MGLevelT<T>& lv, unsigned n) {
  const unsigned t = n / (unsigned)lv.Nx;
  const unsigned k = t / (unsigned)lv.Ny;
  return {(int)(n - t * (unsigned)lv.Nx), (int)(t - k * (unsigned)lv.Ny), (int)k};
}
template <typename T>
__device__ __forceinline__ bool on_boundary(const MGLevelT<T>& lv, const MGNode& q) {
  return on_boundary(q.i, q.j, q.k, lv.Nx, lv.Ny, lv.Nz);
}

// The eight entries of an element's matrix on unit coefficient, by the axes along which
// its two nodes differ (bit 0: x, 1: y, 2: z): 1D k = [1 -1; -1 1] / h, m = [2 1; 1 2] h / 6.
template <typename T>
struct Q1Entries {
  T k[8];
  __host__ __device__ explicit Q1Entries(const T (&entries)[8]) {
    for (int o = 0; o < 8; ++o) k[o] = entries[o];
  }
  template <typename Level>
  __host__ __device__ explicit Q1Entries(const Level& lv) {
    const T kx[2] = {T(1.0 / lv.hx), T(-1.0 / lv.hx)}, ky[2] = {T(1.0 / lv.hy), T(-1.0 / lv.hy)},
            kz[2] = {T(1.0 / lv.hz), T(-1.0 / lv.hz)};
    const T mx[2] = {T(lv.hx / 3.0), T(lv.hx / 6.0)}, my[2] = {T(lv.hy / 3.0), T(lv.hy / 6.0)},
            mz[2] = {T(lv.hz / 3.0), T(lv.hz / 6.0)};
    for (int o = 0; o < 8; ++o) {
      const int x = o & 1, y = (o >> 1) & 1, z = o >> 2;
      k[o] = kx[x] * my[y] * mz[z] + mx[x] * ky[y] * mz[z] + mx[x] * my[y] * kz[z];
    }
  }
};

// (A_l x) at an interior node of a Q1 level from the 8 elements' coefficients and the 27
// nodes' values: the coefficients of the elements between the
// node and each neighbour summed first (4 for a face neighbour, 2 for an edge, 1 for a
// corner), the neighbours of one class then times that class's matrix entry.  x is zero on
// the boundary (every vector of the coarse levels is).
template <typename T>
__device__ __forceinline__ T q1_stencil(const Q1Entries<T>& K, const T (&c)[2][2][2], const T (&xs)[3][3][3]) {
  // edge sums (two elements), face sums (four), all eight
  T zy[2][2], zx[2][2], yx[2][2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      zy[u][v] = c[u][v][0] + c[u][v][1];
      zx[u][v] = c[u][0][v] + c[u][1][v];
      yx[u][v] = c[0][u][v] + c[1][u][v];
    }
  const T fz[2] = {zy[0][0] + zy[0][1], zy[1][0] + zy[1][1]};
  const T fy[2] = {zy[0][0] + zy[1][0], zy[0][1] + zy[1][1]};
  const T fx[2] = {zx[0][0] + zx[1][0], zx[0][1] + zx[1][1]};
  T acc = K.k[0] * ((fz[0] + fz[1]) * xs[1][1][1]);
  acc = fma(K.k[1], fma(fx[0], xs[1][1][0], fx[1] * xs[1][1][2]), acc);
  acc = fma(K.k[2], fma(fy[0], xs[1][0][1], fy[1] * xs[1][2][1]), acc);
  acc = fma(K.k[4], fma(fz[0], xs[0][1][1], fz[1] * xs[2][1][1]), acc);
  T s3 = T(0), s5 = T(0), s6 = T(0), s7 = T(0);
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      s3 = fma(yx[u][v], xs[1][2 * u][2 * v], s3);
      s5 = fma(zx[u][v], xs[2 * u][1][2 * v], s5);
      s6 = fma(zy[u][v], xs[2 * u][2 * v][1], s6);
      s7 = fma(c[u][v][0], xs[2 * u][2 * v][0], s7);
      s7 = fma(c[u][v][1], xs[2 * u][2 * v][2], s7);
    }
  acc = fma(K.k[3], s3, acc);
  acc = fma(K.k[5], s5, acc);
  acc = fma(K.k[6], s6, acc);
  return fma(K.k[7], s7, acc);
}
template <typename T>
__device__ __forceinline__ T q1_apply_at(const MGLevelT<T>& lv, const Q1Entries<T>& K, const T* x,
                                         unsigned n, const MGNode& q) {
  const unsigned sy = (unsigned)lv.Nx, sz = sy * (unsigned)lv.Ny;
  const unsigned e0 = (unsigned)(q.i - 1) + (unsigned)lv.nx * ((unsigned)(q.j - 1) + (unsigned)lv.ny * (unsigned)(q.k - 1));
  T c[2][2][2];
#pragma unroll
  for (int z = 0; z < 2; ++z)
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int w = 0; w < 2; ++w)
        c[z][y][w] = lv.coef[e0 + w + (unsigned)lv.nx * (y + (unsigned)lv.ny * z)];
  T xs[3][3][3];
  const T* const x0 = x + (n - 1u - sy - sz);
#pragma unroll
  for (int z = 0; z < 3; ++z)
#pragma unroll
    for (int y = 0; y < 3; ++y)
#pragma unroll
      for (int w = 0; w < 3; ++w) xs[z][y][w] = x0[w + sy * y + sz * z];
  return q1_stencil(K, c, xs);
}
// the same at any node (identity on the boundary)
template <typename T>
__device__ __forceinline__ T q1_row(const MGLevelT<T>& lv, const Q1Entries<T>& K, const T* x, unsigned n) {
  const MGNode q = node_at(lv, n);
  return on_boundary(lv, q) ? x[n] : q1_apply_at(lv, K, x, n, q);
}

template <typename T>
__global__ void __launch_bounds__(256) k_q1_apply(MGLevelT<T> lv, Q1Entries<T> K, const T* __restrict__ x,
                                                  T* __restrict__ y) {
  const unsigned n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < (unsigned)lv.nodes) y[n] = q1_row(lv, K, x, n);
}
// The operator passes of a Chebyshev-Jacobi smoother of a Q1 level (the arithmetic of
// k_cheb_start / k_cheb_step / k_cheb_finish around k_q1_apply; at degree 1 the products
// rounded on their own, as those kernels store them, so that no contraction changes a bit);
// the modes are HmChebMode's, z the result of the last step
template <typename T, int MODE>
__global__ void __launch_bounds__(256) k_q1_cheb(MGLevelT<T> lv, Q1Entries<T> K, const T* __restrict__ b,
                                                 const T* __restrict__ in, T* x, T* r, T* __restrict__ dout,
                                                 T* z, int k, int first, int last) {
  const unsigned n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (unsigned)lv.nodes) return;
  const T t = q1_row(lv, K, in, n);
  if constexpr (MODE == CH_RESIDUAL) {
    r[n] = b[n] - t;
  } else if constexpr (MODE == CH_STEP1) {
    z[n] = in[n] + mul_rn(T(1.0 / lv.cheb[0]) * (b[n] - t), lv.idiag[n]);
  } else if constexpr (MODE == CH_START) {
    const T ri = b[n] - t;
    r[n] = ri;
    dout[n] = T(1.0 / lv.cheb[0]) * ri * lv.idiag[n];
  } else {
    const T di = in[n];
    const T ri = (first ? b[n] : r[n]) - t;
    const T xi = first ? di : x[n] + di;
    const T dn = fma(T(lv.cheb[1 + k]), di, T(lv.cheb[1 + kChebMax + k]) * ri * lv.idiag[n]);
    if (last == 2) {
      z[n] = xi + dn;
    } else {
      x[n] = xi;
      r[n] = ri;
      if (last == 0) dout[n] = dn;
    }
  }
}

__global__ void k_q1_diag(MGLevel lv, double* __restrict__ diag) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= lv.nodes) return;
  const int i = (int)(n % lv.Nx);
  const int64_t t = n / lv.Nx;
  const int j = (int)(t % lv.Ny), k = (int)(t / lv.Ny);
  if (on_boundary(i, j, k, lv.Nx, lv.Ny, lv.Nz)) { diag[n] = 1.0; return; }
  const double kaa = (1.0 / lv.hx) * (lv.hy / 3.0) * (lv.hz / 3.0) +
                     (lv.hx / 3.0) * (1.0 / lv.hy) * (lv.hz / 3.0) +
                     (lv.hx / 3.0) * (lv.hy / 3.0) * (1.0 / lv.hz);
  double c = 0.0;
  for (int e3 = 0; e3 < 2; ++e3)
    for (int e2 = 0; e2 < 2; ++e2)
      for (int e1 = 0; e1 < 2; ++e1)
        c += lv.coef[(i - 1 + e1) + (int64_t)lv.nx * ((j - 1 + e2) + (int64_t)lv.ny * (k - 1 + e3))];
  diag[n] = c * kaa;
}

// level-1 coefficients: sum_q D(q) / |e| (D = w|J| e^m in the operator's layout)
__global__ void k_coef_from_q2(Lattice L, int pitch, const double* __restrict__ Dq, double inv_vol,
                               double* __restrict__ coef) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= L.ne) return;
  const int64_t row = e / L.nx, rows = (int64_t)L.ny * L.nz;
  const double* const D = Dq + row * pitch + (e - row * L.nx);
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < 27; ++q) s += D[(int64_t)q * rows * pitch];
  coef[e] = s * inv_vol;
}

__global__ void k_recip(int64_t n, const double* __restrict__ a, double* __restrict__ ia) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) ia[i] = 1.0 / a[i];
}

// a coarse element's coefficient: the mean of its 8 children
__global__ void k_coef_coarsen(MGLevel f, MGLevel c, const double* __restrict__ cf,
                               double* __restrict__ cc) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= c.elems) return;
  const int ex = (int)(e % c.nx);
  const int64_t t = e / c.nx;
  const int ey = (int)(t % c.ny), ez = (int)(t / c.ny);
  double s = 0.0;
  for (int z = 0; z < 2; ++z)
    for (int y = 0; y < 2; ++y)
      for (int x = 0; x < 2; ++x)
        s += cf[(2 * ex + x) + (int64_t)f.nx * ((2 * ey + y) + (int64_t)f.ny * (2 * ez + z))];
  cc[e] = 0.125 * s;
}

// b_c = R r_f (full weighting, the transpose of trilinear interpolation); 0 on the
// coarse boundary
template <typename T>
__device__ __forceinline__ T restrict_at(const MGLevelT<T>& f, const MGLevelT<T>& c, const T* rf,
                                         unsigned n) {
  const MGNode q = node_at(c, n);
  if (on_boundary(c, q)) return T(0);
  const unsigned sy = (unsigned)f.Nx, sz = sy * (unsigned)f.Ny;
  const T* const r0 = rf + ((unsigned)(2 * q.i - 1) + sy * (unsigned)(2 * q.j - 1) + sz * (unsigned)(2 * q.k - 1));
  T s = T(0);
#pragma unroll
  for (int dk = 0; dk < 3; ++dk)
#pragma unroll
    for (int dj = 0; dj < 3; ++dj) {
      const T* const r = r0 + sy * dj + sz * dk;
      const T w = T((dj == 1 ? 1.0 : 0.5) * (dk == 1 ? 1.0 : 0.5));
      s = fma(w, fma(T(0.5), r[0] + r[2], r[1]), s);
    }
  return s;
}
// b_c = R r_f and, given d, the smoother's first direction d = b idiag / theta
template <typename T>
__global__ void __launch_bounds__(256) k_restrict(MGLevelT<T> f, MGLevelT<T> c, const T* __restrict__ rf,
                                                  T* __restrict__ bc, T* __restrict__ d) {
  const unsigned n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (unsigned)c.nodes) return;
  const T b = restrict_at(f, c, rf, n);
  bc[n] = b;
  if (d != nullptr) d[n] = mul_rn(T(1.0 / c.cheb[0]) * b, c.idiag[n]);
}

// P x_c (trilinear) at the fine nodes 2q, 2q + 1 along each axis of the coarse cell at q;
// v[x + 2 y + 4 z]
template <typename T>
__device__ __forceinline__ void prolong_cell(const MGLevelT<T>& c, const T* xc, unsigned nc, T (&v)[8]) {
  const unsigned sy = (unsigned)c.Nx, sz = sy * (unsigned)c.Ny;
  T e[2][2][2];
#pragma unroll
  for (int z = 0; z < 2; ++z)
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const T a = xc[nc + sy * y + sz * z], b = xc[nc + 1u + sy * y + sz * z];
      e[z][y][0] = a;
      e[z][y][1] = T(0.5) * (a + b);
    }
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const T y0 = e[0][0][x], y1 = T(0.5) * (e[0][0][x] + e[0][1][x]);
    const T z0 = e[1][0][x], z1 = T(0.5) * (e[1][0][x] + e[1][1][x]);
    v[x] = y0;
    v[2 + x] = y1;
    v[4 + x] = T(0.5) * (y0 + z0);
    v[6 + x] = T(0.5) * (y1 + z1);
  }
}
// x_f += P x_c on the coarse cell number m (a thread's 8 fine nodes; a fine node on the
// boundary is left alone)
template <typename T>
__device__ __forceinline__ void prolong_add_cell(const MGLevelT<T>& f, const MGLevelT<T>& c, const T* xc,
                                                 T* xf, unsigned m) {
  const unsigned cx = (unsigned)c.Nx - 1u, cy = (unsigned)c.Ny - 1u;
  const unsigned t = m / cx, i = m - t * cx, k = t / cy, j = t - k * cy;
  T v[8];
  prolong_cell(c, xc, i + (unsigned)c.Nx * (j + (unsigned)c.Ny * k), v);
  const unsigned n0 = 2u * i + (unsigned)f.Nx * (2u * j + (unsigned)f.Ny * 2u * k);
#pragma unroll
  for (int h = 0; h < 8; ++h) {
    if ((!(h & 1) && i == 0) || (!(h & 2) && j == 0) || (!(h & 4) && k == 0)) continue;
    const unsigned n = n0 + (h & 1) + (unsigned)f.Nx * (((h >> 1) & 1) + (unsigned)f.Ny * (h >> 2));
    xf[n] += v[h];
  }
}
template <typename T>
HM_HD unsigned coarse_cells(const MGLevelT<T>& c) {
  return (unsigned)(c.Nx - 1) * (unsigned)(c.Ny - 1) * (unsigned)(c.Nz - 1);
}
template <typename T>
__global__ void __launch_bounds__(256) k_prolong_add(MGLevelT<T> f, MGLevelT<T> c, const T* __restrict__ xc,
                                                     T* __restrict__ xf) {
  const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < coarse_cells(c)) prolong_add_cell(f, c, xc, xf, m);
}

// Chebyshev-Jacobi (idiag: the reciprocal of the Jacobi diagonal): start (r = b - t, or
// r = b with t == nullptr; d = r idiag / theta; x = 0 when zero_x), step (x += d; r -= t;
// d = c1 d + c2 r idiag unless last), finish (x += d)
template <typename T>
__global__ void k_cheb_start(int64_t n, const T* __restrict__ b, const T* __restrict__ t,
                             const T* __restrict__ idiag, const double* __restrict__ cheb,
                             int zero_x, T* __restrict__ x, T* __restrict__ r,
                             T* __restrict__ d) {
  const T inv_theta = T(1.0 / cheb[0]);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T ri = t ? b[i] - t[i] : b[i];
    r[i] = ri;
    d[i] = inv_theta * ri * idiag[i];
    if (zero_x) x[i] = T(0);
  }
}
template <typename T>
__global__ void k_cheb_step(int64_t n, T* __restrict__ x, T* __restrict__ d,
                            T* __restrict__ r, const T* __restrict__ t,
                            const T* __restrict__ idiag, const double* __restrict__ cheb,
                            int k, int last) {
  const T c1 = T(cheb[1 + k]), c2 = T(cheb[1 + kChebMax + k]);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T di = d[i];
    x[i] += di;
    const T ri = r[i] - t[i];
    r[i] = ri;
    if (!last) d[i] = fma(c1, di, c2 * ri * idiag[i]);
  }
}
template <typename T>
__global__ void k_cheb_finish(int64_t n, T* __restrict__ x, const T* __restrict__ d) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] += d[i];
}

// ---- exact solve of a small coarsest level
// Interior node q of a level <-> (1 + q % (Nx-2), 1 + (q / (Nx-2)) % (Ny-2), ...).
constexpr int kCoarseDirectMax = 64;
template <typename T>
__device__ __forceinline__ int64_t interior_node(const MGLevelT<T>& lv, int q) {
  const int ax = lv.Nx - 2, ay = lv.Ny - 2;
  return (1 + q % ax) + (int64_t)lv.Nx * ((1 + (q / ax) % ay) + (int64_t)lv.Ny * (1 + q / (ax * ay)));
}
template <typename T>
__host__ __device__ inline int interior_count(const MGLevelT<T>& lv) {
  return (lv.Nx - 2) * (lv.Ny - 2) * (lv.Nz - 2);
}
// set-up (one CTA): the interior block column by column (the operator on unit vectors in
// lv.t), then its inverse by Gauss-Jordan elimination (SPD: no pivoting), into lv.cinv
__global__ void __launch_bounds__(256) k_coarse_factor(MGLevel lv) {
  __shared__ double A[kCoarseDirectMax][kCoarseDirectMax + 1];
  const int n = interior_count(lv);
  const int tid = threadIdx.x, nt = blockDim.x;
  const Q1Entries<double> K(lv);
  for (int64_t i = tid; i < lv.nodes; i += nt) lv.t[i] = 0.0;
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    if (tid == 0) lv.t[interior_node(lv, j)] = 1.0;
    __syncthreads();
    for (int i = tid; i < n; i += nt) A[i][j] = q1_row(lv, K, lv.t, (unsigned)interior_node(lv, i));
    __syncthreads();
    if (tid == 0) lv.t[interior_node(lv, j)] = 0.0;
    __syncthreads();
  }
  for (int k = 0; k < n; ++k) {
    const double p = A[k][k];
    __syncthreads();
    if (tid == 0) A[k][k] = 1.0;
    __syncthreads();
    for (int j = tid; j < n; j += nt) A[k][j] = A[k][j] / p;
    __syncthreads();
    for (int e = tid; e < n * n; e += nt) {
      const int i = e / n, j = e % n;
      if (i != k && j != k) A[i][j] = fma(-A[i][k], A[k][j], A[i][j]);
    }
    __syncthreads();
    for (int i = tid; i < n; i += nt)
      if (i != k) A[i][k] = -A[i][k] * A[k][k];
    __syncthreads();
  }
  for (int e = tid; e < n * n; e += nt) lv.cinv[e] = A[e / n][e % n];
}
// x = A_l^{-1} b for the small coarsest level, inside one CTA (x zero on the boundary)
template <typename T>
__device__ void coarse_direct(const MGLevelT<T>& lv, const T* __restrict__ b, T* __restrict__ x) {
  const int n = interior_count(lv);
  for (int64_t i = threadIdx.x; i < lv.nodes; i += blockDim.x) x[i] = T(0);
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    T acc = T(0);
    for (int j = 0; j < n; ++j) acc = fma(lv.cinv[i * n + j], b[interior_node(lv, j)], acc);
    x[interior_node(lv, i)] = acc;
  }
  __syncthreads();
}
template <typename T>
__global__ void __launch_bounds__(256) k_coarse_solve(MGLevelT<T> lv, const T* __restrict__ b,
                                                      T* __restrict__ x) {
  coarse_direct(lv, b, x);
}

// ---- the coarse levels of a cycle in one cluster
// Launched level by level, a coarse level costs four launches (eight at degree 2) of a few
// microseconds each, almost all latency.  One cluster of CTAs runs the whole part of the
// V-cycle from the restriction into its first level to that level's result, node for node the
// same arithmetic but for the exact coarse solve (a warp sums a row by shuffles).  Its vectors live in the CTAs' shared memory: a level's node
// planes are dealt out in slabs, a CTA computes its own planes and reads its neighbours'
// through the cluster's shared memory, and a cluster barrier stands where the launches
// were; coefficients and reciprocal diagonals are copied in at the start.  The levels of at
// most kSoloNodes nodes lie in the first CTA alone, between block barriers.  Measured
// (FP64, degree 1): 28 us for the levels 17^3, 9^3, 5^3, 3^3 of 32^3 and 64^3, 19 us for
// 13^3, 7^3, 4^3, against ~47 and ~39 us as launches with one CTA from 1000 nodes down.  A
// 33^3 level in the cluster takes 44 us more and ~16 us as launches.  An iteration with the
// cluster from the level named down, against from the level below it: 17^3 73.6 us and 82.4
// (16^3 elements), 21^3 76.6 and 84.9, 25x17x21 134 and 143, 25^3 89 and 92 (48^3: 165 and
// 175), 29^3 125 and 123, 31x27x23 225 and 223 -- kTailNodes could lie at 16,000; it was set
// between 17^3 and 33^3.  A level of 9^3 in one CTA takes 3 us more than in the cluster.
constexpr int kTailMax = 8;
constexpr int64_t kTailNodes = 5000;
constexpr int64_t kSoloNodes = 150, kTailMost = 1 << 20;
constexpr int kTailThreads = 512;
constexpr int kTailBytes = 216 * 1024;       // shared memory of a CTA at most
enum TailVec { TV_B = 0, TV_X = 1, TV_R = 2, TV_D = 3, TV_E = 4 };   // D, E: degree > 1
template <typename T>
struct TailLevel {
  int nx, ny, Nx, Ny, Nz;
  int A, ppc;            // nodes of a plane, planes per CTA
  int tab;               // first entry of the level in the plane table
  int off, vs;           // the first vector's place in the pool, from one vector to the next
  int idiag_at, coef_at; // places of the reciprocal diagonal and the coefficients
  int degree;
  T entries[8];          // Q1Entries
  const T* coef;
  const T* idiag;
  const T* cinv;
  const double* cheb;
};
template <typename T>
struct MGTail {
  MGLevelT<T> fine;      // the level above: its r is restricted
  TailLevel<T> lv[kTailMax];
  T* out;                // the first level's result
  int count, solo;           // levels, the first of those in one CTA alone
  int planes, pool;          // entries of the plane table, reals of the pool
};
// the layout for clusters of `ctas`; false: it does not fit
template <typename T>
bool plan_tail(const MGLevelT<T>* lvs, int first, int nlev, int ctas, MGTail<T>* t) {
  t->count = nlev - first;
  if (t->count < 1 || t->count > kTailMax) return false;
  t->planes = t->pool = 0;
  t->solo = t->count;
  auto take = [&](int n) { const int at = t->pool; t->pool += n; return at; };
  for (int q = 0; q < t->count; ++q) {
    const MGLevelT<T>& l = lvs[first + q];
    TailLevel<T>& v = t->lv[q];
    if (l.nodes > kTailMost) return false;
    if (l.nodes <= kSoloNodes && t->solo == t->count) t->solo = q;
    v.nx = l.nx; v.ny = l.ny; v.Nx = l.Nx; v.Ny = l.Ny; v.Nz = l.Nz;
    const Q1Entries<T> K(l);
    for (int o = 0; o < 8; ++o) v.entries[o] = K.k[o];
    v.A = l.Nx * l.Ny;
    v.ppc = q >= t->solo ? l.Nz : (l.Nz + ctas - 1) / ctas;
    v.tab = t->planes;
    t->planes += l.Nz;
    v.vs = v.ppc * v.A;
    // degree 1 needs three vectors, more and a Chebyshev coarse solve five
    v.off = take(v.vs * (l.degree == 1 ? 3 : 5));
    v.idiag_at = take(v.vs);
    v.coef_at = take((v.ppc + 1) * l.nx * l.ny);
    v.degree = l.degree;
    v.coef = l.coef; v.idiag = l.idiag; v.cinv = l.cinv; v.cheb = l.cheb;
  }
  return 8 * (int64_t)t->planes + (int64_t)sizeof(T) * t->pool <= kTailBytes;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// this CTA's shared memory address p, in CTA `rank` of the cluster (generic addresses)
template <typename T>
__device__ __forceinline__ T* in_cta(T* p, unsigned rank) {
  uint64_t q;
  asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
  return reinterpret_cast<T*>(q);
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

template <typename T>
struct TailView {
  const TailLevel<T>& l;
  T* const* planes;      // the level's plane table
  const T* idiag;        // of the own planes
  const T* coef;         // of the element planes from k0 - 1 on
  int k0, k1;            // own planes
  Q1Entries<T> K;
  const T* cheb;         // 1 / theta, then c1, c2 of step q at [2 q - 1], [2 q]
  __device__ __forceinline__ TailView(const TailLevel<T>& lev, T* const* tab, T* pool, unsigned rank, const T* ch)
      : l(lev), planes(tab + lev.tab), idiag(pool + lev.idiag_at), coef(pool + lev.coef_at),
        k0(min((int)rank * lev.ppc, lev.Nz)), k1(min(((int)rank + 1) * lev.ppc, lev.Nz)), K(lev.entries), cheb(ch) {}
  __device__ __forceinline__ T* plane(int v, int k) const { return planes[k] + v * l.vs; }
  __device__ __forceinline__ void sync() const {
    if (l.ppc == l.Nz) __syncthreads();
    else cluster_sync();
  }
  // f(k, i, j, o, s): every own node, o its place in its plane, s in the own planes
  template <typename F>
  __device__ __forceinline__ void each(F f) const {
    const unsigned n = (unsigned)(max(0, k1 - k0) * l.A);
    for (unsigned s = threadIdx.x; s < n; s += blockDim.x) {
      const unsigned kl = s / (unsigned)l.A, o = s - kl * (unsigned)l.A, j = o / (unsigned)l.Nx;
      f(k0 + (int)kl, (int)(o - j * (unsigned)l.Nx), (int)j, (int)o, (int)s);
    }
  }
  __device__ __forceinline__ bool boundary(int i, int j, int k) const {
    return on_boundary(i, j, k, l.Nx, l.Ny, l.Nz);
  }
  // (A x) at a node, x the vector v
  __device__ __forceinline__ T row(int v, int k, int i, int j, int o) const {
    const T* const p = plane(v, k);
    if (boundary(i, j, k)) return p[o];
    const T* const c0 = coef + ((i - 1) + l.nx * ((j - 1) + l.ny * (k - k0)));   // element plane k - 1
    T c[2][2][2];
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int w = 0; w < 2; ++w) c[z][y][w] = c0[w + l.nx * (y + l.ny * z)];
    const T* const pl[3] = {plane(v, k - 1) + o, p + o, plane(v, k + 1) + o};
    T xs[3][3][3];
#pragma unroll
    for (int z = 0; z < 3; ++z)
#pragma unroll
      for (int y = 0; y < 3; ++y)
#pragma unroll
        for (int w = 0; w < 3; ++w) xs[z][y][w] = pl[z][(w - 1) + l.Nx * (y - 1)];
    return q1_stencil(K, c, xs);
  }
};

// Chebyshev smoothing from zero: B and the first direction (X at degree 1, else D) given;
// the result in X, with want_r its residual in R
template <typename T>
__device__ void tail_smooth_zero(const TailView<T>& V, bool want_r, int degree) {
  if (degree == 1 && V.l.degree == 1) {
    if (!want_r) return;
    V.each([&](int k, int i, int j, int o, int) {
      V.plane(TV_R, k)[o] = V.plane(TV_B, k)[o] - V.row(TV_X, k, i, j, o);
    });
    V.sync();
    return;
  }
  int in = TV_D, out = TV_E;
  for (int q = 1; q <= degree; ++q) {
    const bool last = q == degree, first = q == 1;
    const T c1 = V.cheb[2 * q - 1], c2 = V.cheb[2 * q];
    V.each([&](int k, int i, int j, int o, int s) {
      const T di = V.plane(in, k)[o];
      T* const x = V.plane(TV_X, k) + o;
      *x = first ? di : *x + di;
      if (last && !want_r) return;
      const T ri = (first ? V.plane(TV_B, k)[o] : V.plane(TV_R, k)[o]) - V.row(in, k, i, j, o);
      V.plane(TV_R, k)[o] = ri;
      if (!last) V.plane(out, k)[o] = fma(c1, di, c2 * ri * V.idiag[s]);
    });
    V.sync();
    const int t = in; in = out; out = t;
  }
}
// the same from X; the result in R at degree 1, else in X, or in out (global memory)
template <typename T>
__device__ void tail_smooth_x(const TailView<T>& V, T* gout) {
  const T inv_theta = V.cheb[0];
  const int degree = V.l.degree;
  if (degree == 1) {
    V.each([&](int k, int i, int j, int o, int s) {
      const T xn = V.plane(TV_X, k)[o] +
                   mul_rn(inv_theta * (V.plane(TV_B, k)[o] - V.row(TV_X, k, i, j, o)), V.idiag[s]);
      if (gout != nullptr) gout[(unsigned)k * (unsigned)V.l.A + (unsigned)o] = xn;
      else V.plane(TV_R, k)[o] = xn;
    });
    V.sync();
    return;
  }
  V.each([&](int k, int i, int j, int o, int s) {
    const T ri = V.plane(TV_B, k)[o] - V.row(TV_X, k, i, j, o);
    V.plane(TV_R, k)[o] = ri;
    V.plane(TV_D, k)[o] = inv_theta * ri * V.idiag[s];
  });
  V.sync();
  int in = TV_D, out = TV_E;
  for (int q = 1; q < degree; ++q) {
    const T c1 = V.cheb[2 * q - 1], c2 = V.cheb[2 * q];
    const bool last = q + 1 == degree;
    V.each([&](int k, int i, int j, int o, int s) {
      const T di = V.plane(in, k)[o];
      const T ri = V.plane(TV_R, k)[o] - V.row(in, k, i, j, o);
      T* const x = V.plane(TV_X, k) + o;
      const T dn = fma(c1, di, c2 * ri * V.idiag[s]);
      const T xi = last ? (*x + di) + dn : *x + di;
      V.plane(TV_R, k)[o] = ri;
      V.plane(out, k)[o] = dn;
      if (last && gout != nullptr) gout[(unsigned)k * (unsigned)V.l.A + (unsigned)o] = xi;
      else *x = xi;
    });
    V.sync();
    const int t = in; in = out; out = t;
  }
}

template <typename R>
__global__ void __launch_bounds__(kTailThreads) k_mg_tail(const __grid_constant__ MGTail<R> T) {
  extern __shared__ __align__(16) unsigned char tail_smem[];
  __shared__ R coeffs[kTailMax][2 * kChebMax];
  R** const tab = reinterpret_cast<R**>(tail_smem);
  R* const pool = reinterpret_cast<R*>(tail_smem + 8 * T.planes);
  const unsigned rank = cluster_rank();
  // the plane table, coefficients and reciprocal diagonals
  for (int q = 0; q < T.count; ++q) {
    const TailLevel<R>& l = T.lv[q];
    for (int k = threadIdx.x; k < l.Nz; k += blockDim.x) {
      const unsigned owner = (unsigned)k / (unsigned)l.ppc;
      R* const p = pool + l.off + (k - (int)owner * l.ppc) * l.A;
      tab[l.tab + k] = owner == rank ? p : in_cta(p, owner);
    }
    for (int i = threadIdx.x; i <= 2 * l.degree; i += blockDim.x)
      coeffs[q][i] = i == 0 ? R(1.0 / l.cheb[0]) : R(l.cheb[(i & 1) ? 1 + (i + 1) / 2 : 1 + kChebMax + i / 2]);
    const int k0 = min((int)rank * l.ppc, l.Nz), k1 = min(((int)rank + 1) * l.ppc, l.Nz);
    for (int i = threadIdx.x; i < (k1 - k0) * l.A; i += blockDim.x)
      pool[l.idiag_at + i] = l.idiag[(unsigned)k0 * (unsigned)l.A + (unsigned)i];
    const int ea = l.nx * l.ny;
    const int e0 = max(k0 - 1, 0), e1 = min(k1, l.Nz - 1);       // element planes
    for (int i = threadIdx.x; i < (e1 - e0) * ea; i += blockDim.x)
      pool[l.coef_at + (e0 - (k0 - 1)) * ea + i] = l.coef[(unsigned)e0 * (unsigned)ea + (unsigned)i];
  }
  cluster_sync();
  auto down = [&](int q) {   // restriction (from global memory, then from R), smoothing
    const TailView<R> V(T.lv[q], tab, pool, rank, coeffs[q]);
    const R inv_theta = V.cheb[0];
    const bool coarsest = q + 1 == T.count;
    const int first = V.l.degree == 1 ? TV_X : TV_D;
    const TailLevel<R>& fl = T.lv[q > 0 ? q - 1 : 0];
    V.each([&](int k, int i, int j, int o, int s) {
      R b = R(0);
      if (!V.boundary(i, j, k)) {
        const int fx = q == 0 ? T.fine.Nx : fl.Nx, fa = q == 0 ? fx * T.fine.Ny : fl.A;
        const int f0 = (2 * i - 1) + fx * (2 * j - 1);
#pragma unroll
        for (int dk = 0; dk < 3; ++dk) {
          const int fk = 2 * k - 1 + dk;
          const R* const rp = (q == 0 ? T.fine.r + (size_t)fk * fa : tab[fl.tab + fk] + TV_R * fl.vs) + f0;
#pragma unroll
          for (int dj = 0; dj < 3; ++dj) {
            const R* const r = rp + fx * dj;
            b = fma(R((dj == 1 ? 1.0 : 0.5) * (dk == 1 ? 1.0 : 0.5)), fma(R(0.5), r[0] + r[2], r[1]), b);
          }
        }
      }
      V.plane(TV_B, k)[o] = b;
      if (coarsest && V.l.cinv != nullptr) V.plane(TV_X, k)[o] = R(0);
      else V.plane(first, k)[o] = mul_rn(inv_theta * b, V.idiag[s]);
    });
    V.sync();
    if (!coarsest) {
      tail_smooth_zero(V, true, V.l.degree);
    } else if (V.l.cinv == nullptr) {
      tail_smooth_zero(V, false, V.l.degree);
    } else {
      // the exact solve: a warp per row of the inverse, by the first CTA
      const int ax = V.l.Nx - 2, ay = V.l.Ny - 2, n = ax * ay * (V.l.Nz - 2);
      auto at = [&](int v, int m) -> R* {
        return V.plane(v, 1 + m / (ax * ay)) + (1 + m % ax) + V.l.Nx * (1 + (m / ax) % ay);
      };
      if (rank == 0)
        for (int i = threadIdx.x >> 5; i < n; i += blockDim.x >> 5) {
          R acc = R(0);
          for (int c = threadIdx.x & 31; c < n; c += 32) acc = fma(V.l.cinv[i * n + c], *at(TV_B, c), acc);
#pragma unroll
          for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
          if ((threadIdx.x & 31) == 0) *at(TV_X, i) = acc;
        }
      V.sync();
    }
    if (coarsest && q == 0)
      V.each([&](int k, int, int, int o, int) {
        T.out[(unsigned)k * (unsigned)V.l.A + (unsigned)o] = V.plane(TV_X, k)[o];
      });
  };
  auto up = [&](int q) {     // prolongation, smoothing
    const TailView<R> V(T.lv[q], tab, pool, rank, coeffs[q]);
    const TailLevel<R>& c = T.lv[q + 1];
    const int cv = q + 2 == T.count || c.degree != 1 ? TV_X : TV_R;
    V.each([&](int k, int i, int j, int o, int) {
      if (V.boundary(i, j, k)) return;
      R v[2];
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        const R* const p = tab[c.tab + ((k + z) >> 1)] + cv * c.vs;
        const R* const p0 = p + c.Nx * (j >> 1);
        const R* const p1 = p + c.Nx * ((j + 1) >> 1);
        const int a0 = i >> 1, a1 = (i + 1) >> 1;
        v[z] = R(0.5) * (R(0.5) * (p0[a0] + p0[a1]) + R(0.5) * (p1[a0] + p1[a1]));
      }
      V.plane(TV_X, k)[o] += R(0.5) * (v[0] + v[1]);
    });
    V.sync();
    tail_smooth_x(V, q == 0 ? T.out : nullptr);
  };
  for (int q = 0; q < T.solo; ++q) down(q);
  if (rank == 0) {
    for (int q = T.solo; q < T.count; ++q) down(q);
    for (int q = T.count - 2; q >= T.solo; --q) up(q);
  }
  if (T.solo > 0) cluster_sync();
  for (int q = min(T.solo, T.count - 1) - 1; q >= 0; --q) up(q);
  cluster_sync();        // no CTA leaves while another reads its shared memory
}

// set-up: a deterministic pseudo-random start vector (0 on the boundary)
__global__ void k_mg_seed(MGLevel lv, double* __restrict__ v) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= lv.nodes) return;
  const int i = (int)(n % lv.Nx);
  const int64_t t = n / lv.Nx;
  const int j = (int)(t % lv.Ny), k = (int)(t / lv.Ny);
  uint64_t h = (uint64_t)n * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
  h ^= h >> 31; h *= 0xBF58476D1CE4E5B9ull; h ^= h >> 29;
  v[n] = on_boundary(i, j, k, lv.Nx, lv.Ny, lv.Nz) ? 0.0 : (double)(h >> 11) * 0x1.0p-53 - 0.5;
}
// A step of the power iteration on a Q1 level, y = D^-1 A x (0 on the boundary)
__global__ void __launch_bounds__(256) k_q1_power(MGLevel lv, Q1Entries<double> K, const double* __restrict__ x,
                                                  double* __restrict__ y) {
  const unsigned n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < (unsigned)lv.nodes) y[n] = q1_row(lv, K, x, n) * lv.idiag[n];
}
// The Rayleigh quotient lambda = v.w / v.diag.v of w = A v, and from it the Chebyshev
// coefficients of the interval [hi / lo_div, hi], hi = 1.1 lambda (the last block; lambda
// is 0 where the quotient is not defined).  part holds two sums a block.
__global__ void __launch_bounds__(256) k_mg_interval(int64_t n, const double* __restrict__ v,
                                                     const double* __restrict__ w,
                                                     const double* __restrict__ diag, double* __restrict__ part,
                                                     unsigned* __restrict__ counter, double lo_div, int degree,
                                                     double* __restrict__ cheb) {
  __shared__ double sh[32];
  double a = 0.0, b = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double vi = v[i];
    a = fma(vi, w[i], a);
    b = fma(vi * diag[i], vi, b);
  }
  a = block_sum(a, sh);
  b = block_sum(b, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = a;
    part[gridDim.x + blockIdx.x] = b;
  }
  if (!last_block(counter)) return;
  a = b = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
    a += __ldcg(part + i);
    b += __ldcg(part + gridDim.x + i);
  }
  a = block_sum(a, sh);
  b = block_sum(b, sh);
  if (threadIdx.x != 0) return;
  *counter = 0u;
  const double lambda = b > 0.0 && isfinite(a / b) ? a / b : 0.0;
  const double hi = 1.1 * lambda, lo = hi / lo_div;
  const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
  double rho_old = 1.0 / sigma;
  cheb[0] = theta;
  for (int k = 1; k <= degree && k < kChebMax; ++k) {
    const double rho = 1.0 / (2.0 * sigma - rho_old);
    cheb[1 + k] = rho * rho_old;
    cheb[1 + kChebMax + k] = 2.0 * rho / delta;
    rho_old = rho;
  }
}

}  // namespace hm

using namespace hm;

namespace {
inline cudaStream_t S_(void* s) { return reinterpret_cast<cudaStream_t>(s); }
inline int blocks_for(int64_t n) { return (int)((n + 255) / 256); }

// the levels of the cycle in precision T
template <typename T> MGLevelT<T>* levels_of(hm_mg* mg);
template <> MGLevelT<double>* levels_of<double>(hm_mg* mg) { return mg->lv; }
template <> MGLevelT<float>* levels_of<float>(hm_mg* mg) { return mg->lv32; }

// clean: x is zero on the Dirichlet nodes (the level-0 operator pass then skips
// the markers); every vector of a cycle is when its right-hand side is
template <typename T>
int apply_level(hm_mg* mg, int l, const T* x, T* y, bool clean, cudaStream_t s) {
  if (l == 0) {
    if constexpr (std::is_same<T, double>::value) {
      if (clean) return hm_launch_apply_A_clean(mg->L, mg->jac, mg->ess, x, y, (void*)s);
      return hm_launch_apply_A(mg->L, mg->jac, HM_FP64, mg->ess, x, y, (void*)s);
    } else {
      return hm_launch_apply_A32(mg->L, mg->jac32, mg->ess, x, y, clean, (void*)s);
    }
  }
  const MGLevelT<T>& lv = levels_of<T>(mg)[l];
  k_q1_apply<T><<<blocks_for(lv.nodes), 256, 0, s>>>(lv, Q1Entries<T>(lv), x, y);
  return HM_OK;
}

// Chebyshev smoothing of A_l x = b: from x = 0 (zero_x) or from the given x; with
// want_r the residual b - A x of the result is left in lv.r
template <typename T>
int smooth(hm_mg* mg, int l, const T* b, T* x, bool zero_x, bool want_r, int degree,
           bool clean, cudaStream_t s) {
  MGLevelT<T>& lv = levels_of<T>(mg)[l];
  int rc;
  const int g = kMGBlocks;
  if (zero_x) {
    k_cheb_start<T><<<g, 256, 0, s>>>(lv.nodes, b, nullptr, lv.idiag, lv.cheb, 1, x, lv.r, lv.d);
  } else {
    if ((rc = apply_level<T>(mg, l, x, lv.t, clean, s))) return rc;
    k_cheb_start<T><<<g, 256, 0, s>>>(lv.nodes, b, lv.t, lv.idiag, lv.cheb, 0, x, lv.r, lv.d);
  }
  for (int k = 1; k <= degree; ++k) {
    const bool last = k == degree;
    if (last && !want_r) {
      k_cheb_finish<T><<<g, 256, 0, s>>>(lv.nodes, x, lv.d);
      break;
    }
    if ((rc = apply_level<T>(mg, l, lv.d, lv.t, clean, s))) return rc;
    k_cheb_step<T><<<g, 256, 0, s>>>(lv.nodes, x, lv.d, lv.r, lv.t, lv.idiag, lv.cheb, k, last ? 1 : 0);
  }
  return HM_OK;
}

// CTAs of a tail cluster on the current device (found once): 16 where the device holds such
// a cluster, else the portable 8
template <typename T>
int tail_ctas() {
  static std::atomic<int> most[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = most[dev].load();
  if (n == 0) {
    if (cudaFuncSetAttribute(k_mg_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailBytes) != cudaSuccess)
      return 0;
    n = 8;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 16; at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = kTailBytes;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int active = 0;
    if (cudaFuncSetAttribute(k_mg_tail<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&active, k_mg_tail<T>, &cfg) == cudaSuccess && active >= 1)
      n = 16;
    (void)cudaGetLastError();
    most[dev].store(n);
  }
  return n;
}
// the tail from level mg->tail_first, the residual of the level above restricted first;
// the result in that level's x
template <typename T>
int launch_tail(hm_mg* mg, cudaStream_t s) {
  MGLevelT<T>* lvs = levels_of<T>(mg);
  const int l = mg->tail_first, n = tail_ctas<T>();
  MGTail<T> TL{};
  if (n == 0 || !plan_tail<T>(lvs, l, mg->nlev, n, &TL)) return HM_ERR_CUDA;
  TL.fine = lvs[l - 1];
  TL.out = lvs[l].x;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = n; at.val.clusterDim.y = at.val.clusterDim.z = 1;
  if (TL.solo == 0) at.val.clusterDim.x = 1;
  cfg.gridDim = dim3(at.val.clusterDim.x);
  cfg.blockDim = dim3(kTailThreads);
  cfg.dynamicSmemBytes = 8 * (size_t)TL.planes + sizeof(T) * (size_t)TL.pool;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_mg_tail<T>, TL) == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

template <typename T>
int vcycle(hm_mg* mg, int l, const T* b, T* x, bool clean, cudaStream_t s, T** out);
// the coarse correction of level l: its residual lv.r restricted and the cycle of level
// l + 1; *xc: where its result lies
template <typename T>
int coarse_cycle(hm_mg* mg, int l, bool clean, cudaStream_t s, T** xc) {
  MGLevelT<T>* lvs = levels_of<T>(mg);
  MGLevelT<T>& cv = lvs[l + 1];
  if (l + 1 == mg->tail_first) {
    *xc = cv.x;
    return launch_tail<T>(mg, s);
  }
  // with fused smoothing the first direction is formed here (at degree 1 into the iterate)
  T* const d = !mg->fused || cv.cinv ? nullptr : cv.degree == 1 ? cv.x : cv.d;
  k_restrict<T><<<blocks_for(cv.nodes), 256, 0, s>>>(lvs[l], cv, lvs[l].r, cv.b, d);
  return vcycle<T>(mg, l + 1, cv.b, cv.x, clean, s, xc);
}

// fused smoothing of a Q1 level from zero, its first direction given (coarse_cycle): the
// result in x, with want_r its residual in r
template <typename T>
void q1_smooth_zero(const MGLevelT<T>& lv, bool want_r, cudaStream_t s) {
  const Q1Entries<T> K(lv);
  const int g = blocks_for(lv.nodes), degree = lv.degree;
  if (degree == 1) {
    if (want_r)
      k_q1_cheb<T, CH_RESIDUAL><<<g, 256, 0, s>>>(lv, K, lv.b, lv.x, nullptr, lv.r, nullptr, nullptr, 0, 0, 0);
    return;
  }
  T* in = lv.d;
  T* out = lv.t;
  const int steps = want_r ? degree : degree - 1;
  for (int k = 1; k <= steps; ++k) {
    k_q1_cheb<T, CH_NEXT><<<g, 256, 0, s>>>(lv, K, lv.b, in, lv.x, lv.r, out, lv.x, k, k == 1,
                                            k < steps ? 0 : want_r ? 1 : 2);
    T* const t = in; in = out; out = t;
  }
}
// fused smoothing from x; returns where the result lies
template <typename T>
T* q1_smooth_x(const MGLevelT<T>& lv, cudaStream_t s) {
  const Q1Entries<T> K(lv);
  const int g = blocks_for(lv.nodes), degree = lv.degree;
  if (degree == 1) {
    k_q1_cheb<T, CH_STEP1><<<g, 256, 0, s>>>(lv, K, lv.b, lv.x, nullptr, nullptr, nullptr, lv.t, 0, 0, 0);
    return lv.t;
  }
  k_q1_cheb<T, CH_START><<<g, 256, 0, s>>>(lv, K, lv.b, lv.x, nullptr, lv.r, lv.d, nullptr, 0, 0, 0);
  T* in = lv.d;
  T* out = lv.t;
  for (int k = 1; k < degree; ++k) {
    k_q1_cheb<T, CH_NEXT><<<g, 256, 0, s>>>(lv, K, lv.b, in, lv.x, lv.r, out, lv.x, k, 0, k + 1 < degree ? 0 : 2);
    T* const t = in; in = out; out = t;
  }
  return lv.x;
}

// The V-cycle from level l for A_l x = b.  *out: where the result lies -- x, except
// for a Q1 level whose fused post-smoothing writes it to the level's lv.t.  The fused
// passes of level 0 are level0_cycle's.
template <typename T>
int vcycle(hm_mg* mg, int l, const T* b, T* x, bool clean, cudaStream_t s, T** out) {
  int rc;
  *out = x;
  MGLevelT<T>* lvs = levels_of<T>(mg);
  MGLevelT<T>& lv = lvs[l];
  const bool fuse = mg->fused && l > 0;
  if (l == mg->nlev - 1) {
    if (lv.cinv) {
      k_coarse_solve<T><<<1, 256, 0, s>>>(lv, b, x);
      return HM_OK;
    }
    if (fuse && lv.degree > 1) {
      q1_smooth_zero(lv, false, s);
      return HM_OK;
    }
    return smooth<T>(mg, l, b, x, true, false, mg->coarse_degree, clean, s);
  }
  MGLevelT<T>& cv = lvs[l + 1];
  if (fuse) q1_smooth_zero(lv, true, s);
  else if ((rc = smooth<T>(mg, l, b, x, true, true, mg->degree, clean, s))) return rc;
  T* xc = nullptr;
  if ((rc = coarse_cycle<T>(mg, l, clean, s, &xc))) return rc;
  k_prolong_add<T><<<blocks_for(coarse_cells(cv)), 256, 0, s>>>(lv, cv, xc, x);
  if (fuse) {
    *out = q1_smooth_x(lv, s);
    return HM_OK;
  }
  return smooth<T>(mg, l, b, x, false, false, mg->degree, clean, s);
}

// z = V(r) inside the solves (every vector zero on the Dirichlet nodes) with the level-0
// smoothing fused into its operator passes: the first direction is given (hm_mg_first_dir),
// the passes read r and write z themselves, in FP32 too
bool level0_fused(const hm_mg* mg) { return mg->fused && mg->nlev > 1; }
template <typename T>
int level0_cycle(hm_mg* mg, const double* r, double* z, cudaStream_t s, double* fail, HmBeta* beta) {
  MGLevelT<T>& lv = levels_of<T>(mg)[0];
  const MGLevel& l0 = mg->lv[0];
  constexpr bool kFP64 = std::is_same<T, double>::value;
  const int degree = mg->degree;
  void* const jac = kFP64 ? mg->jac : (void*)mg->jac32;
  HmCheb<T> c{};
  c.b = r; c.idiag = l0.idiag; c.cheb = l0.cheb; c.fail = fail;
  c.r = lv.r;
  // the iterate: at degree 1 beside z (the last pass reads its neighbours), FP64 at higher
  // degrees z itself
  T* d = lv.t;
  T* e = lv.d;
  if constexpr (kFP64) c.x = degree == 1 ? lv.t : z;
  else c.x = degree == 1 ? (d = lv.x) : lv.x;
  int rc;
  if (degree == 1) {
    c.mode = CH_RESIDUAL;
    c.in = c.x;
    if ((rc = hm_launch_cheb<T>(mg->L, jac, mg->ess, c, (void*)s))) return rc;
  } else {
    c.mode = CH_NEXT;
    for (int k = 1; k <= degree; ++k) {
      c.k = k; c.first = k == 1; c.last = k == degree ? 1 : 0;
      c.in = d; c.dout = e;
      if ((rc = hm_launch_cheb<T>(mg->L, jac, mg->ess, c, (void*)s))) return rc;
      T* const t = d; d = e; e = t;
    }
  }
  T* xc = nullptr;
  if ((rc = coarse_cycle<T>(mg, 0, true, s, &xc))) return rc;
  MGLevelT<T>& cv = levels_of<T>(mg)[1];
  k_prolong_add<T><<<blocks_for(coarse_cells(cv)), 256, 0, s>>>(lv, cv, xc, c.x);
  c.first = 0;
  c.in = c.x;
  c.z = z;
  c.beta = beta;
  if (degree == 1) {
    c.mode = CH_STEP1;
    return hm_launch_cheb<T>(mg->L, jac, mg->ess, c, (void*)s);
  }
  d = lv.t;
  e = lv.d;
  c.mode = CH_START;
  c.dout = d;
  if ((rc = hm_launch_cheb<T>(mg->L, jac, mg->ess, c, (void*)s))) return rc;
  c.mode = CH_NEXT;
  for (int k = 1; k < degree; ++k) {
    c.k = k; c.last = k + 1 == degree ? 2 : 0;
    c.in = d; c.dout = e;
    if ((rc = hm_launch_cheb<T>(mg->L, jac, mg->ess, c, (void*)s))) return rc;
    T* const t = d; d = e; e = t;
  }
  return HM_OK;
}

__global__ void k_to_float(int64_t n, const double* __restrict__ a, float* __restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}
// rows of nx entries from one pitch to another
__global__ void k_jac_to_float(int64_t rows, int nx, int pa, int pb, const double* __restrict__ a,
                               float* __restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows * nx;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / nx, c = i - r * nx;
    b[r * pb + c] = (float)a[r * pa + c];
  }
}
__global__ void k_to_double(int64_t n, const float* __restrict__ a, double* __restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (double)a[i];
}

// z = V(r) with the cycle in FP32, step by step on level 0: r rounded to FP32 first, the
// result widened at the end
int vcycle_single(hm_mg* mg, const double* r, double* z, bool clean, cudaStream_t s) {
  MGLevelT<float>* lv = mg->lv32;
  k_to_float<<<kMGBlocks, 256, 0, s>>>(lv[0].nodes, r, lv[0].b);
  float* out = nullptr;
  const int rc = vcycle<float>(mg, 0, lv[0].b, lv[0].x, clean, s, &out);
  if (rc) return rc;
  k_to_double<<<kMGBlocks, 256, 0, s>>>(lv[0].nodes, out, z);
  return HM_OK;
}

// the tail: the Q1 levels (l >= 1) of at most max_nodes nodes that fit a cluster's shared
// memory (in FP64), at most kTailMax of them (max_nodes = 0: none)
void set_tail(hm_mg* mg, int64_t max_nodes) {
  mg->tail_nodes = max_nodes;
  mg->tail_first = mg->nlev;
  const int n = tail_ctas<double>();
  if (n == 0 || tail_ctas<float>() != n) return;
  MGTail<double> t;
  for (int l = mg->nlev - 1; l >= 1 && mg->lv[l].nodes <= max_nodes && plan_tail(mg->lv, l, mg->nlev, n, &t); --l)
    mg->tail_first = l;
}

// the level hierarchy of a lattice (no memory touched)
int plan_levels(const Lattice& L, MGLevel* lv, int max_levels) {
  int nl = 0;
  MGLevel z{};
  z.nx = L.nx; z.ny = L.ny; z.nz = L.nz;
  z.Nx = L.Nx; z.Ny = L.Ny; z.Nz = L.Nz;
  z.hx = L.hx; z.hy = L.hy; z.hz = L.hz;
  z.nodes = L.ndof; z.elems = L.ne;
  lv[nl++] = z;
  MGLevel q = z;                       // Q1 on the same elements
  q.Nx = L.nx + 1; q.Ny = L.ny + 1; q.Nz = L.nz + 1;
  q.nodes = (int64_t)q.Nx * q.Ny * q.Nz;
  if (L.nx < 2 || L.ny < 2 || L.nz < 2) return nl;
  lv[nl++] = q;
  while (nl < max_levels) {
    const MGLevel& f = lv[nl - 1];
    if ((f.nx & 1) || (f.ny & 1) || (f.nz & 1) || f.nx < 4 || f.ny < 4 || f.nz < 4) break;
    MGLevel c{};
    c.nx = f.nx / 2; c.ny = f.ny / 2; c.nz = f.nz / 2;
    c.Nx = c.nx + 1; c.Ny = c.ny + 1; c.Nz = c.nz + 1;
    c.hx = 2 * f.hx; c.hy = 2 * f.hy; c.hz = 2 * f.hz;
    c.nodes = (int64_t)c.Nx * c.Ny * c.Nz;
    c.elems = (int64_t)c.nx * c.ny * c.nz;
    lv[nl++] = c;
  }
  return nl;
}

// the coarsest level is solved exactly (through its inverse) when it is a Q1 level with
// few interior nodes
bool exact_coarsest(const hm_mg* mg, int l) {
  if (mg->nlev < 2 || l != mg->nlev - 1) return false;
  const int ni = interior_count(mg->lv[l]);
  return ni >= 1 && ni <= kCoarseDirectMax;
}

// the FP32 copies of the level data on work32 (in floats; each piece starts on 128 bytes)
int64_t layout_single(hm_mg* mg, float* work32) {
  float* w = work32;
  int64_t used = 0;
  auto take = [&](int64_t n) {
    const int64_t m = (n + 31) / 32 * 32;
    float* p = w ? w + used : nullptr;
    used += m;
    return p;
  };
  const Lattice& L = mg->L;
  float* jac = take(54 * L.ne);
  if (work32) mg->jac32 = jac;
  for (int l = 0; l < mg->nlev; ++l) {
    const MGLevel& d = mg->lv[l];
    MGLevelT<float> f{};
    f.nx = d.nx; f.ny = d.ny; f.nz = d.nz;
    f.Nx = d.Nx; f.Ny = d.Ny; f.Nz = d.Nz;
    f.hx = d.hx; f.hy = d.hy; f.hz = d.hz;
    f.nodes = d.nodes; f.elems = d.elems;
    f.coef = l >= 1 ? take(d.elems) : nullptr;
    f.diag = nullptr;
    f.idiag = take(d.nodes);
    f.x = take(d.nodes); f.b = take(d.nodes); f.r = take(d.nodes);
    f.d = take(d.nodes); f.t = take(d.nodes);
    f.cinv = exact_coarsest(mg, l) ? take(kCoarseDirectMax * kCoarseDirectMax) : nullptr;
    f.cheb = d.cheb;
    f.degree = d.degree;
    if (work32) mg->lv32[l] = f;
  }
  return used;
}

// the FP32 level data from the FP64 set-up (the point's D, coefficients, reciprocal
// diagonals, the coarse inverse; the Chebyshev coefficients are shared)
void refresh_single(hm_mg* mg, cudaStream_t s) {
  const Lattice& L = mg->L;
  k_jac_to_float<<<4 * kMGBlocks, 256, 0, s>>>(27 * (int64_t)L.ny * L.nz, L.nx, hm_jac_pitch(L, HM_FP64),
                                               hm_jac_pitch(L, HM_FP32),
                                               static_cast<const double*>(mg->jac), mg->jac32);
  for (int l = 0; l < mg->nlev; ++l) {
    const MGLevel& d = mg->lv[l];
    MGLevelT<float>& f = mg->lv32[l];
    f.degree = d.degree;
    k_to_float<<<kMGBlocks, 256, 0, s>>>(d.nodes, d.idiag, f.idiag);
    if (l >= 1) k_to_float<<<kMGBlocks, 256, 0, s>>>(d.elems, d.coef, f.coef);
    if (d.cinv) {
      const int ni = interior_count(d);
      k_to_float<<<1, 256, 0, s>>>((int64_t)ni * ni, d.cinv, f.cinv);
    }
  }
}

__global__ void k_count_mismatch(Lattice L, const uint8_t* __restrict__ ess, unsigned* __restrict__ bad) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= L.ndof) return;
  const int i = (int)(n % L.Nx);
  const int64_t t = n / L.Nx;
  const int j = (int)(t % L.Ny), k = (int)(t / L.Ny);
  const bool b = on_boundary(i, j, k, L.Nx, L.Ny, L.Nz);
  if ((ess != nullptr && ess[n] != 0) != b) atomicAdd(bad, 1u);
}
}  // namespace

// inside the MG-PCG, whose residuals are zero on the Dirichlet nodes
int hm_mg_vcycle(hm_mg* mg, const double* r, double* z, void* stream, double* fail, HmBeta* beta) {
  cudaStream_t s = S_(stream);
  if (level0_fused(mg))
    return mg->single ? level0_cycle<float>(mg, r, z, s, fail, beta) : level0_cycle<double>(mg, r, z, s, fail, beta);
  if (mg->single) return vcycle_single(mg, r, z, true, s);
  double* out = nullptr;
  return vcycle<double>(mg, 0, r, z, true, s, &out);
}
// the buffer and operands of the level-0 smoother's first direction, where the cycle inside
// the solves takes it ready made
HmFirstDir hm_mg_first_dir(const hm_mg* mg) {
  HmFirstDir f{};
  if (!level0_fused(mg)) return f;
  f.idiag = mg->lv[0].idiag;
  f.cheb = mg->lv[0].cheb;
  if (mg->single) f.d32 = mg->degree == 1 ? mg->lv32[0].x : mg->lv32[0].t;
  else f.d64 = mg->lv[0].t;
  return f;
}
bool hm_mg_flexible(const hm_mg* mg) { return mg->single != 0; }
const double* hm_mg_level0_diag(const hm_mg* mg) { return mg->lv[0].diag; }
void* hm_mg_jac(const hm_mg* mg) { return mg->jac; }
const uint8_t* hm_mg_ess(const hm_mg* mg) { return mg->ess; }
const hm::Lattice* hm_mg_lattice(const hm_mg* mg) { return &mg->L; }

extern "C" int64_t hm_mg_workspace_bytes(const hm_lattice* h) {
  const Lattice* L = hm_lattice_geometry(h);
  if (!L) return 0;
  MGLevel lv[16];
  const int nl = plan_levels(*L, lv, 16);
  int64_t doubles = 4 * L->ndof + 3 * kMGBlocks + 64 + nl * (2 * kChebMax + 8) +
                    kCoarseDirectMax * kCoarseDirectMax + 8;
  for (int l = 1; l < nl; ++l) doubles += lv[l].elems + 7 * lv[l].nodes + 8;
  return doubles * (int64_t)sizeof(double);
}

extern "C" int hm_mg_create(const hm_lattice* h, void* work, int degree, int coarse_degree,
                            hm_mg** out) {
  const Lattice* L = hm_lattice_geometry(h);
  if (!L || !work || !out || degree < 1 || degree >= kChebMax || coarse_degree < 1 ||
      coarse_degree >= kChebMax)
    return HM_ERR_ARG;
  hm_mg* mg = new (std::nothrow) hm_mg();
  if (!mg) return HM_ERR_NOMEM;
  mg->L = *L;
  mg->degree = degree;
  mg->coarse_degree = coarse_degree;
  mg->nlev = plan_levels(*L, mg->lv, 16);
  for (int l = 0; l < mg->nlev; ++l) mg->lv[l].degree = l == mg->nlev - 1 ? coarse_degree : degree;
  mg->fused = 1;
  mg->single = 0;
  mg->jac32 = nullptr;
  double* w = static_cast<double*>(work);
  auto take = [&](int64_t n) { double* p = w; w += n; return p; };
  mg->scratch = take(3 * kMGBlocks + 64);
  mg->checked_ess = nullptr;
  for (int l = 0; l < mg->nlev; ++l) mg->lv[l].cheb = take(2 * kChebMax + 8);
  MGLevel& z = mg->lv[0];
  z.r = take(L->ndof); z.d = take(L->ndof); z.t = take(L->ndof); z.idiag = take(L->ndof);
  z.x = z.b = nullptr; z.coef = nullptr; z.diag = nullptr;
  for (int l = 1; l < mg->nlev; ++l) {
    MGLevel& lv = mg->lv[l];
    lv.coef = take(lv.elems);
    lv.diag = take(lv.nodes);
    lv.idiag = take(lv.nodes);
    lv.x = take(lv.nodes); lv.b = take(lv.nodes); lv.r = take(lv.nodes);
    lv.d = take(lv.nodes); lv.t = take(lv.nodes);
    lv.cinv = nullptr;
    w += 8;
  }
  z.cinv = nullptr;
  // an exact coarse solve when the coarsest Q1 level has few interior nodes
  if (exact_coarsest(mg, mg->nlev - 1))
    mg->lv[mg->nlev - 1].cinv = take(kCoarseDirectMax * kCoarseDirectMax);
  set_tail(mg, kTailNodes);
  *out = mg;
  return HM_OK;
}

// the point's operator: coefficients, diagonals and eigenvalue bounds, all on the device
// (the first set-up with a marker array checks it: one synchronisation)
extern "C" int hm_mg_setup(hm_mg* mg, void* jac, const uint8_t* ess, const double* diag,
                           void* stream) {
  if (!mg || !jac || !ess || !diag) return HM_ERR_ARG;
  cudaStream_t s = S_(stream);
  const Lattice& L = mg->L;
  // the Dirichlet nodes must be exactly the boundary (checked once per marker array)
  if (ess != mg->checked_ess) {
    unsigned* bad = reinterpret_cast<unsigned*>(mg->scratch + 3 * kMGBlocks + 8);
    if (cudaMemsetAsync(bad, 0, sizeof(unsigned), s) != cudaSuccess) return HM_ERR_CUDA;
    k_count_mismatch<<<blocks_for(L.ndof), 256, 0, s>>>(L, ess, bad);
    unsigned hbad = 0;
    if (cudaMemcpyAsync(&hbad, bad, sizeof(unsigned), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return HM_ERR_CUDA;
    if (hbad != 0) return HM_ERR_UNSUPPORTED;
    mg->checked_ess = ess;
  }
  mg->jac = jac;
  mg->ess = ess;
  mg->lv[0].diag = const_cast<double*>(diag);
  // coefficients and diagonals of the Q1 levels
  if (mg->nlev > 1) {
    MGLevel& q = mg->lv[1];
    k_coef_from_q2<<<blocks_for(L.ne), 256, 0, s>>>(L, hm_jac_pitch(L, HM_FP64),
                                                    static_cast<const double*>(jac),
                                                    1.0 / (L.hx * L.hy * L.hz), q.coef);
    for (int l = 2; l < mg->nlev; ++l)
      k_coef_coarsen<<<blocks_for(mg->lv[l].elems), 256, 0, s>>>(mg->lv[l - 1], mg->lv[l],
                                                                  mg->lv[l - 1].coef, mg->lv[l].coef);
    for (int l = 1; l < mg->nlev; ++l)
      k_q1_diag<<<blocks_for(mg->lv[l].nodes), 256, 0, s>>>(mg->lv[l], mg->lv[l].diag);
  }
  for (int l = 0; l < mg->nlev; ++l)
    k_recip<<<blocks_for(mg->lv[l].nodes), 256, 0, s>>>(mg->lv[l].nodes, mg->lv[l].diag,
                                                        mg->lv[l].idiag);
  // largest eigenvalue of D^{-1} A per level, on the device: nine steps of the power
  // iteration from a fixed start, unscaled (a step grows the vector by the eigenvalue at
  // most, and that is below 27, the most nodes an element couples), each one launch, then
  // the Rayleigh quotient v.Av / v.Dv; smoothing interval [hi/4, hi], the coarsest level's
  // solve on [hi/64, hi].  (With the scaling, and a quotient at each of ten steps, a step
  // took four launches: 2.3 ms of 16.3 of the two forward solves on 64^3 elements.)
  double* part = mg->scratch;
  unsigned* counter = reinterpret_cast<unsigned*>(mg->scratch + 3 * kMGBlocks);
  if (cudaMemsetAsync(counter, 0, sizeof(unsigned), s) != cudaSuccess) return HM_ERR_CUDA;
  for (int l = 0; l < mg->nlev; ++l) {
    MGLevel& lv = mg->lv[l];
    double* v = lv.d;
    double* w = lv.t;
    k_mg_seed<<<blocks_for(lv.nodes), 256, 0, s>>>(lv, v);
    for (int it = 0; it < 9; ++it) {                    // v is zero on the boundary
      if (l == 0) {
        const int rc = hm_launch_power(L, jac, ess, lv.idiag, v, w, stream);
        if (rc) return rc;
      } else {
        k_q1_power<<<blocks_for(lv.nodes), 256, 0, s>>>(lv, Q1Entries<double>(lv), v, w);
      }
      std::swap(v, w);
    }
    const int rc = apply_level(mg, l, v, w, true, s);
    if (rc) return rc;
    const bool coarsest = l == mg->nlev - 1;
    k_mg_interval<<<std::min<int64_t>(blocks_for(lv.nodes), kMGBlocks), 256, 0, s>>>(
        lv.nodes, v, w, lv.diag, part, counter, coarsest ? 64.0 : 4.0, lv.degree, lv.cheb);
    if (coarsest && lv.cinv) k_coarse_factor<<<1, 256, 0, s>>>(lv);
  }
  if (mg->single) refresh_single(mg, s);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

extern "C" int hm_mg_set_tail_nodes(hm_mg* mg, int64_t max_nodes) {
  if (!mg || max_nodes < 0) return HM_ERR_ARG;
  set_tail(mg, max_nodes);
  return HM_OK;
}

extern "C" int64_t hm_mg_single_workspace_bytes(const hm_lattice* h) {
  const Lattice* L = hm_lattice_geometry(h);
  if (!L) return 0;
  hm_mg probe{};
  probe.L = *L;
  probe.nlev = plan_levels(*L, probe.lv, 16);
  return layout_single(&probe, nullptr) * (int64_t)sizeof(float);
}

// the cycle in FP32 on work32 (hm_mg_single_workspace_bytes), or back in FP64 (null);
// after a set-up the FP32 data are formed at once, on stream
extern "C" int hm_mg_set_single(hm_mg* mg, void* work32, void* stream) {
  if (!mg) return HM_ERR_ARG;
  if (work32 == nullptr) {
    mg->single = 0;
    return HM_OK;
  }
  layout_single(mg, static_cast<float*>(work32));
  mg->single = 1;
  if (mg->jac) {
    refresh_single(mg, S_(stream));
    if (cudaGetLastError() != cudaSuccess) return HM_ERR_CUDA;
  }
  return HM_OK;
}

extern "C" int hm_mg_set_fused(hm_mg* mg, int fused) {
  if (!mg) return HM_ERR_ARG;
  mg->fused = fused != 0;
  return HM_OK;
}

extern "C" int hm_mg_apply(hm_mg* mg, const double* r, double* z, void* stream) {
  if (!mg || !r || !z || !mg->jac) return HM_ERR_ARG;
  double* out = nullptr;
  const int rc = mg->single ? vcycle_single(mg, r, z, false, S_(stream))
                            : vcycle<double>(mg, 0, r, z, false, S_(stream), &out);
  if (rc) return rc;
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

extern "C" int hm_mg_levels(const hm_mg* mg) { return mg ? mg->nlev : 0; }

extern "C" int hm_mg_destroy(hm_mg* mg) {
  delete mg;
  return HM_OK;
}
