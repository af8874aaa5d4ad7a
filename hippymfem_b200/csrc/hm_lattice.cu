// Structured-lattice kernels of the Q2 log-conductivity path (sm_100a).
//
//   k_pattern_*     the CSR graph (diagonal first), the entry->slot map and the
//                   transpose map of a Q2 x Q2 block, arithmetically
//   k_quad          pointwise data D, E = D grad u, F = D grad p, W = D grad u.grad p
//   k_extract_D     the matrix-free Jacobian's data (its apply is in hm_apply.cu)
// (the fused assembly k_tile_assemble is in hm_tile.cu)
#include <cstdio>

#include "hm_common.cuh"
#include "hm_internal.h"

namespace hm {

// =============================================================== pattern kernels
__device__ __forceinline__ void node_of(int64_t n, const Lattice& L, int& i, int& j, int& k) {
  i = (int)(n % L.Nx);
  const int64_t t = n / L.Nx;
  j = (int)(t % L.Ny);
  k = (int)(t / L.Ny);
}

// CSR position of column (ci, cj, ck) within row (i, j, k): diagonal first, the rest
// ascending (ascending lexicographic node number = z, then y, then x rank)
__device__ __forceinline__ int pos_in_row(const Lattice& L, int i, int j, int k, int ci,
                                          int cj, int ck) {
  const int n1 = stencil_n(i, L.Nx), n2 = stencil_n(j, L.Ny);
  const int rank = ((ck - stencil_lo(k)) * n2 + (cj - stencil_lo(j))) * n1 + (ci - stencil_lo(i));
  const int kd = ((k - stencil_lo(k)) * n2 + (j - stencil_lo(j))) * n1 + (i - stencil_lo(i));
  return rank == kd ? 0 : (rank < kd ? rank + 1 : rank);
}

__global__ void k_pattern_indptr(Lattice L, int32_t* __restrict__ indptr) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n > L.ndof) return;
  if (n == L.ndof) {
    indptr[n] = (int32_t)(stencil_prefix(L.Nx, L.Nx) * stencil_prefix(L.Ny, L.Ny) *
                          stencil_prefix(L.Nz, L.Nz));
    return;
  }
  int i, j, k;
  node_of(n, L, i, j, k);
  indptr[n] = (int32_t)row_start(L, i, j, k);
}

// one warp per row: the row's columns in CSR order
__global__ void k_pattern_indices(Lattice L, const int32_t* __restrict__ indptr,
                                  int32_t* __restrict__ indices) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= L.ndof) return;
  int i, j, k;
  node_of(row, L, i, j, k);
  const int n1 = stencil_n(i, L.Nx), n2 = stencil_n(j, L.Ny), n3 = stencil_n(k, L.Nz);
  const int lo1 = stencil_lo(i), lo2 = stencil_lo(j), lo3 = stencil_lo(k);
  const int kd = ((k - lo3) * n2 + (j - lo2)) * n1 + (i - lo1);
  const int len = n1 * n2 * n3;
  const int64_t base = indptr[row];
  for (int pos = lane; pos < len; pos += 32) {
    const int rank = pos == 0 ? kd : (pos <= kd ? pos - 1 : pos);
    const int k1 = rank % n1, t = rank / n1, k2 = t % n2, k3 = t / n2;
    indices[base + pos] = (int32_t)((lo1 + k1) + (int64_t)L.Nx * ((lo2 + k2) + (int64_t)L.Ny * (lo3 + k3)));
  }
}

// entry k = (e*27 + a)*27 + b -> CSR position (patternbuild.build_tables' slot)
__global__ void k_pattern_slot(Lattice L, int32_t* __restrict__ slot) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= L.ne * 729) return;
  const int b = (int)(k % 27);
  const int a = (int)((k / 27) % 27);
  const int64_t e = k / 729;
  const int ex = (int)(e % L.nx), ey = (int)((e / L.nx) % L.ny), ez = (int)(e / ((int64_t)L.nx * L.ny));
  const int i = 2 * ex + a % 3, j = 2 * ey + (a / 3) % 3, kk = 2 * ez + a / 9;
  const int ci = 2 * ex + b % 3, cj = 2 * ey + (b / 3) % 3, ck = 2 * ez + b / 9;
  slot[k] = (int32_t)(row_start(L, i, j, kk) + pos_in_row(L, i, j, kk, ci, cj, ck));
}

// tpos[s] = CSR position of (col, row) for entry s = (row, col)
__global__ void k_pattern_tpos(Lattice L, const int32_t* __restrict__ indptr,
                               int32_t* __restrict__ tpos) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= L.ndof) return;
  int i, j, k;
  node_of(row, L, i, j, k);
  const int n1 = stencil_n(i, L.Nx), n2 = stencil_n(j, L.Ny), n3 = stencil_n(k, L.Nz);
  const int lo1 = stencil_lo(i), lo2 = stencil_lo(j), lo3 = stencil_lo(k);
  const int kd = ((k - lo3) * n2 + (j - lo2)) * n1 + (i - lo1);
  const int len = n1 * n2 * n3;
  const int64_t base = indptr[row];
  for (int pos = lane; pos < len; pos += 32) {
    const int rank = pos == 0 ? kd : (pos <= kd ? pos - 1 : pos);
    const int k1 = rank % n1, t = rank / n1, k2 = t % n2, k3 = t / n2;
    const int ci = lo1 + k1, cj = lo2 + k2, ck = lo3 + k3;
    tpos[base + pos] = (int32_t)(row_start(L, ci, cj, ck) + pos_in_row(L, ci, cj, ck, i, j, k));
  }
}

// ============================================================ quadrature data
// One thread per (element, Gauss point), 8 elements per 216-thread block.  Layout:
// quad[e][c][q], c = 0 D, 1-3 E, 4-6 F, 7 W (each element's 216 values contiguous).
// With mhat, D = w|J| e^m mhat: the data of the directional derivative along mhat
// (the second-order products of the assembled vectors, with f = 0).
template <typename real>
__global__ void __launch_bounds__(216) k_quad(Lattice L, const double* __restrict__ u,
                                              const double* __restrict__ m,
                                              const double* __restrict__ p,
                                              const double* __restrict__ mhat,
                                              real* __restrict__ quad,
                                              uint32_t* __restrict__ status) {
  __shared__ real sv[8][4][27];
  const int le = threadIdx.x / 27, q = threadIdx.x % 27;
  const int64_t e = blockIdx.x * 8LL + le;
  const bool live = e < L.ne;
  if (live) {
    const int ex = (int)(e % L.nx), ey = (int)((e / L.nx) % L.ny), ez = (int)(e / ((int64_t)L.nx * L.ny));
    const int a = q;
    const int64_t node = (2 * ex + a % 3) + (int64_t)L.Nx * ((2 * ey + (a / 3) % 3) + (int64_t)L.Ny * (2 * ez + a / 9));
    sv[le][0][a] = (real)u[node];
    sv[le][1][a] = (real)m[node];
    sv[le][2][a] = (real)p[node];
    if (mhat) sv[le][3][a] = (real)mhat[node];
  }
  __syncthreads();
  if (!live) return;
  const int q1 = q % 3, q2 = (q / 3) % 3, q3 = q / 9;
  real b1[3], b2[3], b3[3], d1[3], d2[3], d3[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b1[a] = (real)bq(q1, a); b2[a] = (real)bq(q2, a); b3[a] = (real)bq(q3, a);
    d1[a] = (real)dbq(q1, a); d2[a] = (real)dbq(q2, a); d3[a] = (real)dbq(q3, a);
  }
  real val[3], gx[3], gy[3], gz[3];
#pragma unroll
  for (int f = 0; f < 3; ++f) {
    const real* x = sv[le][f];
    real vb = 0, vx = 0, vy = 0, vz = 0;
#pragma unroll
    for (int a3 = 0; a3 < 3; ++a3) {
      real sbb = 0, sdb = 0, sbd = 0;
#pragma unroll
      for (int a2 = 0; a2 < 3; ++a2) {
        real xb = 0, xd = 0;
#pragma unroll
        for (int a1 = 0; a1 < 3; ++a1) {
          xb = fma(b1[a1], x[a1 + 3 * a2 + 9 * a3], xb);
          xd = fma(d1[a1], x[a1 + 3 * a2 + 9 * a3], xd);
        }
        sbb = fma(b2[a2], xb, sbb);
        sdb = fma(b2[a2], xd, sdb);
        sbd = fma(d2[a2], xb, sbd);
      }
      vb = fma(b3[a3], sbb, vb);
      vx = fma(b3[a3], sdb, vx);
      vy = fma(b3[a3], sbd, vy);
      vz = fma(d3[a3], sbb, vz);
    }
    val[f] = vb;
    gx[f] = vx / (real)L.hx;
    gy[f] = vy / (real)L.hy;
    gz[f] = vz / (real)L.hz;
  }
  const real wdet = (real)(wq(q1) * wq(q2) * wq(q3) * L.hx * L.hy * L.hz);
  real D = wdet * exp(val[1]);
  if (mhat) {
    // mhat at the point (value only)
    const real* x = sv[le][3];
    real vb = 0;
#pragma unroll
    for (int a3 = 0; a3 < 3; ++a3) {
      real sbb = 0;
#pragma unroll
      for (int a2 = 0; a2 < 3; ++a2) {
        real xb = 0;
#pragma unroll
        for (int a1 = 0; a1 < 3; ++a1) xb = fma(b1[a1], x[a1 + 3 * a2 + 9 * a3], xb);
        sbb = fma(b2[a2], xb, sbb);
      }
      vb = fma(b3[a3], sbb, vb);
    }
    D *= vb;
  }
  const real E[3] = {D * gx[0], D * gy[0], D * gz[0]};
  const real F[3] = {D * gx[2], D * gy[2], D * gz[2]};
  const real W = D * (gx[0] * gx[2] + gy[0] * gy[2] + gz[0] * gz[2]);
  real* out = quad + e * 216;
  out[q] = D;
  out[27 + q] = E[0]; out[54 + q] = E[1]; out[81 + q] = E[2];
  out[108 + q] = F[0]; out[135 + q] = F[1]; out[162 + q] = F[2];
  out[189 + q] = W;
  const bool finite = isfinite(D) && isfinite(E[0]) && isfinite(E[1]) && isfinite(E[2]) &&
                      isfinite(F[0]) && isfinite(F[1]) && isfinite(F[2]) && isfinite(W);
  if (!finite) atomicOr(status, HM_STATUS_NONFINITE);
}

// =============================================== data of the matrix-free Jacobian apply
// D as Dq[q][ez][ey][ex] with rows `pitch` apart (hm_jac_pitch), which the apply
// (hm_apply.cu) reads as TMA boxes
template <typename src, typename real>
__global__ void k_extract_D(Lattice L, int pitch, const src* __restrict__ quad, real* __restrict__ Dq) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= L.ne * 27) return;
  const int64_t e = i / 27;
  const int q = (int)(i - e * 27);
  const int64_t row = e / L.nx;
  Dq[((int64_t)q * L.ny * L.nz + row) * pitch + (e - row * L.nx)] = (real)quad[e * 216 + q];
}

// diagonal of A(D): sum_g D(g) sum_d (d_d phi_n)^2, one thread per node
template <typename real>
__global__ void k_diag_A(Lattice L, const real* __restrict__ quad, const uint8_t* __restrict__ ess,
                         double* __restrict__ diag) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= L.ndof) return;
  const int i = (int)(n % L.Nx), j = (int)((n / L.Nx) % L.Ny), k = (int)(n / ((int64_t)L.Nx * L.Ny));
  if (ess != nullptr && ess[n]) { diag[n] = 1.0; return; }
  const int gi[3] = {i, j, k};
  const int ne[3] = {L.nx, L.ny, L.nz};
  const double h2[3] = {1.0 / (L.hx * L.hx), 1.0 / (L.hy * L.hy), 1.0 / (L.hz * L.hz)};
  // elements touching the node along each axis
  int el0[3], nel[3];
  for (int d = 0; d < 3; ++d) {
    if (gi[d] & 1) { el0[d] = gi[d] / 2; nel[d] = 1; }
    else {
      el0[d] = gi[d] / 2 - 1; nel[d] = 2;
      if (el0[d] < 0) { el0[d] = 0; nel[d] = 1; }
      else if (el0[d] + 1 >= ne[d]) nel[d] = 1;
    }
  }
  double acc = 0.0;
  for (int c3 = 0; c3 < nel[2]; ++c3)
    for (int c2 = 0; c2 < nel[1]; ++c2)
      for (int c1 = 0; c1 < nel[0]; ++c1) {
        const int e1 = el0[0] + c1, e2 = el0[1] + c2, e3 = el0[2] + c3;
        const int a1 = i - 2 * e1, a2 = j - 2 * e2, a3 = k - 2 * e3;
        const real* Dq = quad + (e1 + (int64_t)L.nx * (e2 + (int64_t)L.ny * e3)) * 216;
        // the node's 1D values and derivatives at the three points of each axis, once
        // per element (the products below keep their order)
        double b[3][3], d[3][3];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          b[0][t] = bq(t, a1); b[1][t] = bq(t, a2); b[2][t] = bq(t, a3);
          d[0][t] = dbq(t, a1); d[1][t] = dbq(t, a2); d[2][t] = dbq(t, a3);
        }
#pragma unroll
        for (int q = 0; q < 27; ++q) {
          const int q1 = q % 3, q2 = (q / 3) % 3, q3 = q / 9;
          const double b1 = b[0][q1], b2 = b[1][q2], b3 = b[2][q3];
          const double d1 = d[0][q1], d2 = d[1][q2], d3 = d[2][q3];
          const double s = d1 * d1 * b2 * b2 * b3 * b3 * h2[0] + b1 * b1 * d2 * d2 * b3 * b3 * h2[1] +
                           b1 * b1 * b2 * b2 * d3 * d3 * h2[2];
          acc += (double)Dq[q] * s;
        }
      }
  diag[n] = acc;
}

}  // namespace hm

// ================================================================= host launchers
using namespace hm;

namespace {
inline int grid1(int64_t n, int block) { return (int)((n + block - 1) / block); }
inline cudaStream_t S_(void* s) { return reinterpret_cast<cudaStream_t>(s); }
}

int hm_launch_pattern(const Lattice& L, int32_t* indptr, int32_t* indices, int32_t* slot, void* stream) {
  cudaStream_t s = S_(stream);
  k_pattern_indptr<<<grid1(L.ndof + 1, 256), 256, 0, s>>>(L, indptr);
  if (indices) k_pattern_indices<<<grid1(L.ndof * 32, 256), 256, 0, s>>>(L, indptr, indices);
  if (slot) k_pattern_slot<<<grid1(L.ne * 729, 256), 256, 0, s>>>(L, slot);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

int hm_launch_tpos(const Lattice& L, const int32_t* indptr, int32_t* tpos, void* stream) {
  k_pattern_tpos<<<grid1(L.ndof * 32, 256), 256, 0, S_(stream)>>>(L, indptr, tpos);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

int hm_launch_quad(const Lattice& L, const double* u, const double* m, const double* p,
                   int precision, void* quad, uint32_t* status, void* stream, const double* mhat) {
  const int blocks = grid1(L.ne, 8);
  if (precision == HM_FP32)
    k_quad<float><<<blocks, 216, 0, S_(stream)>>>(L, u, m, p, mhat, (float*)quad, status);
  else
    k_quad<double><<<blocks, 216, 0, S_(stream)>>>(L, u, m, p, mhat, (double*)quad, status);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

int hm_launch_jacobian_prepare(const Lattice& L, const void* quad, int quad_precision, void* jac,
                               int precision, void* stream) {
  const int blocks = grid1(L.ne * 27, 256);
  cudaStream_t s = S_(stream);
  if (quad_precision == HM_FP32) {
    if (precision == HM_FP32) k_extract_D<float, float><<<blocks, 256, 0, s>>>(L, hm_jac_pitch(L, precision), (const float*)quad, (float*)jac);
    else k_extract_D<float, double><<<blocks, 256, 0, s>>>(L, hm_jac_pitch(L, precision), (const float*)quad, (double*)jac);
  } else {
    if (precision == HM_FP32) k_extract_D<double, float><<<blocks, 256, 0, s>>>(L, hm_jac_pitch(L, precision), (const double*)quad, (float*)jac);
    else k_extract_D<double, double><<<blocks, 256, 0, s>>>(L, hm_jac_pitch(L, precision), (const double*)quad, (double*)jac);
  }
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

// x = b on the Dirichlet nodes (the identity rows of the eliminated operator): after it
// every residual of a solve, and so every search direction, is zero there
__global__ void k_ess_take_b(int64_t n, const uint8_t* __restrict__ ess, const double* __restrict__ b,
                             double* __restrict__ x) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n && ess[i]) x[i] = b[i];
}
int hm_launch_ess_take_b(const Lattice& L, const uint8_t* ess, const double* b, double* x,
                         void* stream) {
  if (ess == nullptr) return HM_OK;
  k_ess_take_b<<<grid1(L.ndof, 256), 256, 0, S_(stream)>>>(L.ndof, ess, b, x);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

int hm_launch_diag_A(const Lattice& L, const void* quad, int precision, const uint8_t* ess,
                     double* diag, void* stream) {
  if (precision == HM_FP32)
    k_diag_A<float><<<grid1(L.ndof, 256), 256, 0, S_(stream)>>>(L, (const float*)quad, ess, diag);
  else
    k_diag_A<double><<<grid1(L.ndof, 256), 256, 0, S_(stream)>>>(L, (const double*)quad, ess, diag);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

// ================================================== allocation-free residual / gradient
// A caller that cannot allocate device memory when it needs a residual or a gradient
// (a process whose GPU memory another runtime's pool has already claimed -- JAX/XLA
// preallocates most of the device by default, hypre/MFEM may sit on an Umpire pool --
// or a loop that must not pay for an allocation) gets the assembled vectors through
// hm_lattice_residual_noalloc.  Its one scratch buffer, the pointwise data of the
// lattice's elements, is this fixed array: every GPU that loads the library holds it
// (HM_NOALLOC_MAX_ELEMENTS * 216 doubles, 14.2 MB) until the process exits.
#define HM_NOALLOC_MAX_ELEMENTS 8192
static __device__ __align__(256) double g_noalloc_quad[HM_NOALLOC_MAX_ELEMENTS * 216];

#include <mutex>

namespace {
std::mutex g_noalloc_mutex;
void* g_noalloc_addr[64] = {nullptr};  // device address of g_noalloc_quad, per device
}  // namespace

// The device address of the scratch array on the current device, looked up once per
// device (the array's name is only a host-side stand-in for it).
static int noalloc_scratch(void** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return HM_ERR_CUDA;
  if (dev < 0 || dev >= 64) return HM_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_addr[dev] == nullptr) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_noalloc_quad) != cudaSuccess || ptr == nullptr) return HM_ERR_CUDA;
    g_noalloc_addr[dev] = ptr;
  }
  *out = g_noalloc_addr[dev];
  return HM_OK;
}

extern "C" int hm_lattice_residual_noalloc(const hm_lattice* h, const double* d_u, const double* d_m,
                                           const double* d_p, double f, const uint8_t* d_ess,
                                           double* d_vec_state, double* d_vec_param,
                                           double* d_vec_adjoint, int zero_ess_vectors,
                                           uint32_t* d_status, void* stream) {
  if (!h || !d_u || !d_m || !d_p || !d_status) return HM_ERR_ARG;
  if (!d_vec_state && !d_vec_param && !d_vec_adjoint) return HM_ERR_ARG;
  const hm::Lattice& L = *hm_lattice_geometry(h);
  if (L.ne > HM_NOALLOC_MAX_ELEMENTS) return HM_ERR_NOMEM;
  void* scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  // k_quad overwrites the scratch for every element before the assembly reads it, so
  // nothing is carried over from the previous call
  rc = hm_launch_quad(L, d_u, d_m, d_p, HM_FP64, scratch, d_status, stream);
  if (rc) return rc;
  return hm_launch_assemble(L, scratch, HM_FP64, nullptr, d_ess, f, nullptr, nullptr, nullptr,
                            nullptr, d_vec_state, d_vec_param, d_vec_adjoint, zero_ess_vectors,
                            stream);
}

// ================================================== assembled vectors from the fields
// dR/dp (ADJOINT, with the source -f w|J| phi), dR/du (STATE) and dR/dm (PARAMETER) of the
// point (u, m, p) -- or, with mhat, the second-order products along mhat (D = w|J| e^m
// mhat, f = 0) -- without the pointwise-data array: D at the points, then a pass per vector
// (hm_apply.cu).
namespace hm {
// *same = 0 where (u, m, p) differs from (u0, m0, p0) in any entry (compared as values:
// NaN differs from itself); *same was set nonzero before
__global__ void k_points_compare(int64_t n, const double* __restrict__ u, const double* __restrict__ u0,
                                 const double* __restrict__ m, const double* __restrict__ m0,
                                 const double* __restrict__ p, const double* __restrict__ p0,
                                 uint32_t* __restrict__ same) {
  bool diff = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    diff |= !(u[i] == u0[i]) || !(m[i] == m0[i]) || !(p[i] == p0[i]);
  if (__syncthreads_or(diff) && threadIdx.x == 0) *same = 0u;
}
// out = kept where *same (nonzero), left alone otherwise
__global__ void k_copy_if_same(int64_t n, const uint32_t* __restrict__ same,
                               const double* __restrict__ kept, double* __restrict__ out) {
  if (*same == 0u) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = kept[i];
}
}  // namespace hm

extern "C" int64_t hm_lattice_vectors_workspace_bytes(const hm_lattice* h, int nvectors) {
  if (!h || nvectors < 1 || nvectors > 3) return 0;
  return 8 * 27 * hm_lattice_geometry(h)->ne * (int64_t)nvectors;
}

extern "C" int hm_lattice_vectors(const hm_lattice* h, const double* d_u, const double* d_m,
                                  const double* d_p, const double* d_mhat, double f,
                                  const uint8_t* d_ess, double* d_vec_state, double* d_vec_param,
                                  double* d_vec_adjoint, int zero_ess_vectors, void* d_work,
                                  uint32_t* d_status, void* stream) {
  if (!h || !d_u || !d_m || !d_p || !d_work || !d_status) return HM_ERR_ARG;
  if (!d_vec_state && !d_vec_param && !d_vec_adjoint) return HM_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(d_work) & 7u) != 0) return HM_ERR_ARG;
  const Lattice& L = *hm_lattice_geometry(h);
  double* const outs[3] = {d_vec_adjoint, d_vec_state, d_vec_param};
  const int n = (outs[0] != nullptr) + (outs[1] != nullptr) + (outs[2] != nullptr);
  return hm_launch_vectors(L, d_u, d_m, d_p, d_mhat, f, zero_ess_vectors ? d_ess : nullptr, outs,
                           static_cast<double*>(d_work), 27 * L.ne * n, d_status, nullptr, stream);
}

extern "C" int hm_lattice_vectors_at(const hm_lattice* h, const double* d_u, const double* d_m,
                                     const double* d_p, const double* d_u0, const double* d_m0,
                                     const double* d_p0, const double* d_kept_state,
                                     const double* d_kept_param, const double* d_kept_adjoint,
                                     double f, double* d_vec_state, double* d_vec_param,
                                     double* d_vec_adjoint, void* d_work, uint32_t* d_same,
                                     uint32_t* d_status, void* stream) {
  if (!h || !d_u || !d_m || !d_p || !d_u0 || !d_m0 || !d_p0 || !d_work || !d_same || !d_status)
    return HM_ERR_ARG;
  double* outs[3] = {d_vec_adjoint, d_vec_state, d_vec_param};
  const double* kept[3] = {d_kept_adjoint, d_kept_state, d_kept_param};
  if (!outs[0] && !outs[1] && !outs[2]) return HM_ERR_ARG;
  for (int i = 0; i < 3; ++i)
    if (outs[i] && !kept[i]) return HM_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(d_work) & 7u) != 0) return HM_ERR_ARG;
  const Lattice& L = *hm_lattice_geometry(h);
  cudaStream_t s = S_(stream);
  if (cudaMemsetAsync(d_same, 0xff, sizeof(uint32_t), s) != cudaSuccess) return HM_ERR_CUDA;
  const int cgrid = (int)(grid1(L.ndof, 256) < 148 * 8 ? grid1(L.ndof, 256) : 148 * 8);
  k_points_compare<<<cgrid, 256, 0, s>>>(L.ndof, d_u, d_u0, d_m, d_m0, d_p, d_p0, d_same);
  // the vectors from the fields, every launch standing down when the point is the same
  const int n = (outs[0] != nullptr) + (outs[1] != nullptr) + (outs[2] != nullptr);
  const int rc = hm_launch_vectors(L, d_u, d_m, d_p, nullptr, f, nullptr, outs, static_cast<double*>(d_work),
                                   27 * L.ne * n, d_status, d_same, stream);
  if (rc) return rc;
  for (int i = 0; i < 3; ++i)
    if (outs[i]) k_copy_if_same<<<cgrid, 256, 0, s>>>(L.ndof, d_same, kept[i], outs[i]);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

// ======================================================== boundary mass (Robin term)
// beta * int_{boundary} phi_n phi_c ds added to a block's values in the lattice pattern:
// the boundary-integrator term of the prior's operator (modeling/prior.py:941-944).  On
// the box's face x = 0 the integrand is phi_i(0) phi_ci(0) (= 1 for i = ci = 0) times the
// y and z 1D factors, so each entry gains, per face holding both nodes, the product of
// the two in-face 1D assembled mass entries.  One warp per boundary row.
namespace hm {
// 1D assembled Q2 mass entry between nodes i and c on an axis of n elements of size h
// (3-point Gauss, exact for the products): sum over the elements holding both
__device__ __forceinline__ double mass_1d(int i, int c, int n, double h) {
  const int hi = i > c ? i : c, lo = i < c ? i : c;
  if (hi - lo > 2) return 0.0;
  double s = 0.0;
  for (int e = (hi - 1) / 2 < 0 ? 0 : (hi - 1) / 2; e <= lo / 2 && e < n; ++e) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) t += wq(q) * bq(q, i - 2 * e) * bq(q, c - 2 * e);
    s += h * t;
  }
  return s;
}

__global__ void k_boundary_mass(Lattice L, double beta, double* __restrict__ vals) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= L.ndof) return;
  const int i = (int)(row % L.Nx), j = (int)((row / L.Nx) % L.Ny), k = (int)(row / ((int64_t)L.Nx * L.Ny));
  const bool on[3] = {i == 0 || i == L.Nx - 1, j == 0 || j == L.Ny - 1, k == 0 || k == L.Nz - 1};
  if (!on[0] && !on[1] && !on[2]) return;
  const int n1 = stencil_n(i, L.Nx), n2 = stencil_n(j, L.Ny), n3 = stencil_n(k, L.Nz);
  const int lo1 = stencil_lo(i), lo2 = stencil_lo(j), lo3 = stencil_lo(k);
  const int kd = ((k - lo3) * n2 + (j - lo2)) * n1 + (i - lo1);
  const int len = n1 * n2 * n3;
  const int64_t base = row_start(L, i, j, k);
  for (int pos = lane; pos < len; pos += 32) {
    const int rank = pos == 0 ? kd : (pos <= kd ? pos - 1 : pos);
    const int k1 = rank % n1, t = rank / n1, k2 = t % n2, k3 = t / n2;
    const int c[3] = {lo1 + k1, lo2 + k2, lo3 + k3};
    const int r[3] = {i, j, k};
    double add = 0.0;
    // the faces normal to axis d: the row and the column on the same face
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (!on[d] || c[d] != r[d]) continue;
      const int a = (d + 1) % 3, b = (d + 2) % 3;
      const int na[3] = {L.nx, L.ny, L.nz};
      const double ha[3] = {L.hx, L.hy, L.hz};
      add += mass_1d(r[a], c[a], na[a], ha[a]) * mass_1d(r[b], c[b], na[b], ha[b]);
    }
    if (add != 0.0) vals[base + pos] += beta * add;
  }
}
}  // namespace hm

extern "C" int hm_lattice_add_boundary_mass(const hm_lattice* h, double beta, double* d_vals,
                                            void* stream) {
  if (!h || !d_vals) return HM_ERR_ARG;
  const Lattice& L = *hm_lattice_geometry(h);
  k_boundary_mass<<<grid1(L.ndof * 32, 256), 256, 0, S_(stream)>>>(L, beta, d_vals);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}
