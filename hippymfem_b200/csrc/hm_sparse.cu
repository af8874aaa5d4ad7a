// CSR products, deterministic reductions and the Jacobi-PCG of the incremental solves.
//
// Every reduction is two-pass over a grid fixed by n (reduce_blocks, grid-stride),
// so its summation order depends on n alone: repeated solves are bit-identical.
// The PCG keeps alpha, beta and the residual norms on the device; the host only
// launches and, every check_every iterations, reads one flag.  After convergence the
// step length is frozen at zero, so the result is that of the exact iteration count
// whatever check_every is.
#include <algorithm>
#include <cmath>
#include <new>
#include <type_traits>
#include <vector>

#include "hm_common.cuh"
#include "hm_internal.h"

namespace hm {

constexpr int kReduceBlocks = 1184;  // 8 x 148 SMs, at most
constexpr int kReduceThreads = 256;
// blocks of the vector kernels on n entries (a block with nothing to do still costs its share
// of the reduction: 9.7 against 5 us for the update of 118 k entries)
inline int reduce_blocks(int64_t n) {
  const int64_t b = (n + kReduceThreads - 1) / kReduceThreads;
  return (int)(b < 1 ? 1 : b < kReduceBlocks ? b : kReduceBlocks);
}

// ------------------------------------------------------------------------ SpMV
// G lanes per row (G = 8): a warp covers 4 consecutive rows, which are contiguous in
// the CSR arrays; each group reduces its row with shuffles in a fixed order.  A block takes
// every gridDim.x-th set of 32 rows.  With DOT (a square matrix), also the partial sums of
// x.y, one a block, from which the last block takes the CG step's alpha.
//
// Bound: the values and indices, 12 bytes an entry, once the gathers' latency is hidden: a
// lane has U entries in flight (index, value, then x).  On a 64^3-element lattice (1.6 GB)
// U = 1 took 357 us, 2 379, 4 344, 8 336; on 45 x 52 x 39 125, 118, 107, 104; 32^3 51, 49,
// 45, 45; 24^3 23, 26, 23, 23.  The grid is one wave of resident blocks: with DOT a block's
// reduction then comes once (CG iteration at 24^3, five launches before: 49 -> 41 us, 45 x
// 52 x 39 166 -> 147, 64^3 424 -> 406; with three waves the product alone lost 3 us, with
// one block per 32 rows 4 at 24^3 and 130 at 64^3).
// The transposed product reads its values through tpos, 16 bytes an entry, at scattered
// places; rows that run at the same time have to stay close for the values' lines to be
// shared in L2: one block per 32 rows, 570 us at 64^3 (U = 4; 595 with U = 1, 627 with 8),
// against 690 with 9472 blocks and 876 with 888.
constexpr int kSpmvRows = 32;                          // rows a block covers at a time (256 / G)
constexpr int kSpmvBlocks = 6, kSpmvDotBlocks = 5;     // resident blocks on an SM
template <int G, bool TRANS, bool DOT, int U>
__global__ void __launch_bounds__(256, DOT ? kSpmvDotBlocks : kSpmvBlocks)
    k_spmv(int64_t nrow, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
           const int32_t* __restrict__ tpos, const double* __restrict__ vals,
           const double* __restrict__ x, double* __restrict__ y, double alpha, double beta,
           double* __restrict__ part, double* __restrict__ sc, unsigned* __restrict__ counter) {
  __shared__ double sh[32];
  const int lane = threadIdx.x % G;
  double dot = 0.0;
  for (int64_t r0 = blockIdx.x * (int64_t)(blockDim.x / G); r0 < nrow; r0 += gridDim.x * (int64_t)(blockDim.x / G)) {
    const int64_t row = r0 + threadIdx.x / G;
    double acc = 0.0;
    if (row < nrow) {
      const int b = __ldg(indptr + row), e = __ldg(indptr + row + 1);
      int64_t s = (int64_t)b + lane;
      for (int left = e - b - lane; left > 0; left -= G * U, s += G * U) {
        int col[U];
        double v[U], w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool on = left > u * G;
          col[u] = on ? __ldg(indices + s + u * G) : 0;
          if constexpr (TRANS) v[u] = on ? __ldg(vals + __ldg(tpos + s + u * G)) : 0.0;
          else v[u] = on ? __ldg(vals + s + u * G) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = left > u * G ? __ldg(x + col[u]) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) acc = fma(v[u], w[u], acc);
      }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, G);
    if (row < nrow && lane == 0) {
      const double yn = beta == 0.0 ? alpha * acc : fma(beta, y[row], alpha * acc);
      y[row] = yn;
      if constexpr (DOT) dot = fma(__ldg(x + row), yn, dot);
    }
  }
  if constexpr (DOT) {
    const double t = block_sum(dot, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
    if (last_block(counter)) finish_alpha(part, gridDim.x, sc, counter, sh);
  }
}

__global__ void k_csr_diag(int64_t nrow, const int32_t* __restrict__ indptr,
                           const double* __restrict__ vals, double* __restrict__ diag) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r < nrow) diag[r] = vals[indptr[r]];
}

// ---------------------------------------------------------------- reductions
__global__ void __launch_bounds__(kReduceThreads)
    k_dot_partial(int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                  double* __restrict__ part) {
  __shared__ double sh[32];
  double v = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v = fma(a[i], b[i], v);
  v = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// sum of nq partial arrays part[q * nb + b] -> out[q]
__global__ void k_reduce_final(const double* __restrict__ part, int nb, int nq, double* __restrict__ out) {
  __shared__ double sh[32];
  for (int q = 0; q < nq; ++q) {
    double v = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) v += part[q * nb + b];
    v = block_sum(v, sh);
    if (threadIdx.x == 0) out[q] = v;
  }
}

// ----------------------------------------------------------------------- PCG
// device scalars

// Vector kernels, templated on the vector type T (double, or float for the inner solves
// of the mixed-precision PCG); sums are accumulated in double.

// r = b - q, z = r / diag, p = z; partials of r.z, r.r, b.b
template <typename T>
__global__ void __launch_bounds__(kReduceThreads)
    k_pcg_init(int64_t n, const T* __restrict__ b, const T* __restrict__ q,
               const double* __restrict__ diag, T* __restrict__ r, T* __restrict__ z,
               T* __restrict__ p, double* __restrict__ part) {
  __shared__ double sh[32];
  double rz = 0.0, rr = 0.0, bb = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T ri = b[i] - q[i];
    const T zi = ri / (T)diag[i];
    r[i] = ri; z[i] = zi; p[i] = zi;
    rz = fma((double)ri, (double)zi, rz);
    rr = fma((double)ri, (double)ri, rr);
    bb = fma((double)b[i], (double)b[i], bb);
  }
  rz = block_sum(rz, sh);
  rr = block_sum(rr, sh);
  bb = block_sum(bb, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = rz;
    part[gridDim.x + blockIdx.x] = rr;
    part[2 * gridDim.x + blockIdx.x] = bb;
  }
}

__global__ void k_pcg_init_final(const double* __restrict__ part, int nb, double* __restrict__ sc, double rtol) {
  __shared__ double sh[32];
  double v[3];
  for (int q = 0; q < 3; ++q) {
    double t = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) t += part[q * nb + b];
    v[q] = block_sum(t, sh);
  }
  if (threadIdx.x == 0) {
    sc[SC_RZ] = v[0];
    sc[SC_RR] = v[1];
    sc[SC_BB] = v[2];
    sc[SC_TOL2] = rtol * rtol;
    sc[SC_CONV] = (v[1] <= rtol * rtol * v[2]) ? 0.0 : -1.0;
    sc[SC_IT] = 0.0;
  }
}

// x += alpha p, r -= alpha q, z = r / diag; partials of r.z and r.r; the last
// block to finish takes the step's beta (the iteration count lives on the device, so that
// every batch of iterations launches the same kernels with the same arguments)
template <typename T>
__global__ void __launch_bounds__(kReduceThreads)
    k_pcg_update(int64_t n, double* __restrict__ sc, T* __restrict__ x, T* __restrict__ r,
                 T* __restrict__ z, const T* __restrict__ p, const T* __restrict__ q,
                 const double* __restrict__ diag, double* __restrict__ part,
                 unsigned* __restrict__ counter) {
  __shared__ double sh[32];
  const T alpha = (T)sc[SC_ALPHA];
  double rz = 0.0, rr = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] = fma(alpha, p[i], x[i]);
    const T ri = fma(-alpha, q[i], r[i]);
    const T zi = ri / (T)diag[i];
    r[i] = ri; z[i] = zi;
    rz = fma((double)ri, (double)zi, rz);
    rr = fma((double)ri, (double)ri, rr);
  }
  rz = block_sum(rz, sh);
  rr = block_sum(rr, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = rz;
    part[gridDim.x + blockIdx.x] = rr;
  }
  if (last_block(counter)) {
    double v0 = 0.0, v1 = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
      v0 += __ldcg(part + b);
      v1 += __ldcg(part + gridDim.x + b);
    }
    v0 = block_sum(v0, sh);
    v1 = block_sum(v1, sh);
    if (threadIdx.x == 0) {
      beta_step(v0, v1, sc);
      *counter = 0u;
    }
  }
}

template <typename T>
__global__ void k_pcg_pupdate(int64_t n, const double* __restrict__ sc, const T* __restrict__ z,
                              T* __restrict__ p) {
  if (sc[SC_CONV] >= 0.0) return;
  const T beta = (T)sc[SC_BETA];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = fma(beta, p[i], z[i]);
}

// the multigrid smoother's first direction at a node (the product rounded on its own)
__device__ __forceinline__ void put_first_dir(const HmFirstDir& f, double inv_theta, int64_t i, double r) {
  if (f.d64 != nullptr) f.d64[i] = __dmul_rn(inv_theta * r, f.idiag[i]);
  else if (f.d32 != nullptr) f.d32[i] = (float)__dmul_rn(inv_theta * r, f.idiag[i]);
}

// x += alpha p, r -= alpha q, and the smoother's first direction from r; partials of r.r
// (for a preconditioner applied after it)
// and, given the last preconditioned residual zold, of r.zold (slot 2: the flexible step)
__global__ void __launch_bounds__(kReduceThreads)
    k_pcg_update_rr(int64_t n, const double* __restrict__ sc, double* __restrict__ x,
                    double* __restrict__ r, const double* __restrict__ p,
                    const double* __restrict__ q, double* __restrict__ part, HmFirstDir f,
                    const double* __restrict__ zold = nullptr) {
  __shared__ double sh[32];
  const double alpha = sc[SC_ALPHA];
  const double inv_theta = f.cheb != nullptr ? 1.0 / f.cheb[0] : 0.0;
  double rr = 0.0, rzc = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] = fma(alpha, p[i], x[i]);
    const double ri = fma(-alpha, q[i], r[i]);
    r[i] = ri;
    put_first_dir(f, inv_theta, i, ri);
    rr = fma(ri, ri, rr);
    if (zold != nullptr) rzc = fma(ri, zold[i], rzc);
  }
  rr = block_sum(rr, sh);
  if (threadIdx.x == 0) part[gridDim.x + blockIdx.x] = rr;
  if (zold != nullptr) {
    rzc = block_sum(rzc, sh);
    if (threadIdx.x == 0) part[2 * gridDim.x + blockIdx.x] = rzc;
  }
}

// r = b - q and the smoother's first direction; partials of r.r and b.b (slots 1 and 2)
__global__ void __launch_bounds__(kReduceThreads)
    k_pcg_mg_init(int64_t n, const double* __restrict__ b, const double* __restrict__ q,
                  double* __restrict__ r, double* __restrict__ part, HmFirstDir f) {
  __shared__ double sh[32];
  const double inv_theta = f.cheb != nullptr ? 1.0 / f.cheb[0] : 0.0;
  double rr = 0.0, bb = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double ri = b[i] - q[i];
    r[i] = ri;
    put_first_dir(f, inv_theta, i, ri);
    rr = fma(ri, ri, rr);
    bb = fma(b[i], b[i], bb);
  }
  rr = block_sum(rr, sh);
  bb = block_sum(bb, sh);
  if (threadIdx.x == 0) {
    part[gridDim.x + blockIdx.x] = rr;
    part[2 * gridDim.x + blockIdx.x] = bb;
  }
}

template <typename T>
__global__ void __launch_bounds__(kReduceThreads)
    k_dot_partial_t(int64_t n, const T* __restrict__ a, const T* __restrict__ b, double* __restrict__ part) {
  __shared__ double sh[32];
  double v = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v = fma((double)a[i], (double)b[i], v);
  v = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// Mixed precision (reliable updates): the FP32 vectors are scaled by s, the FP64 norm of
// the residual at the last anchor (sc[SC_S]); sc[SC_SOLD] is the scale before it.
enum { SC_S = SC_TMP0, SC_SOLD = SC_TMP1, SC_TRUE = SC_TMP2 };

// x64 += s x32, x32 = 0
__global__ void k_mx_accum(int64_t n, const double* __restrict__ sc, float* __restrict__ x32,
                           double* __restrict__ x) {
  const double s = sc[SC_S];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] = fma(s, (double)x32[i], x[i]);
    x32[i] = 0.0f;
  }
}

// r64 = b - t64; partials of r64.r64
__global__ void __launch_bounds__(kReduceThreads)
    k_residual64(int64_t n, const double* __restrict__ b, const double* __restrict__ t,
                 const uint8_t* __restrict__ ess, double* __restrict__ r, double* __restrict__ part) {
  __shared__ double sh[32];
  double v = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double ri = (ess && ess[i]) ? 0.0 : b[i] - (t ? t[i] : 0.0);
    r[i] = ri;
    v = fma(ri, ri, v);
  }
  v = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// the true residual's r.r; the new scale
__global__ void k_mx_scale(const double* __restrict__ part, int nb, double* __restrict__ sc) {
  __shared__ double sh[32];
  double t = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) t += part[b];
  t = block_sum(t, sh);
  if (threadIdx.x == 0) {
    sc[SC_TRUE] = t;
    sc[SC_SOLD] = sc[SC_S];
    sc[SC_S] = t > 0.0 ? sqrt(t) : 1.0;
  }
}

// r32 = r64 / s, z32 = r32 / diag, p32 = z32 (reset) or p32 * s_old / s; partials r.z, r.r
__global__ void __launch_bounds__(kReduceThreads)
    k_mx_anchor(int64_t n, const double* __restrict__ r64, const double* __restrict__ diag,
                const double* __restrict__ sc, int reset_p, float* __restrict__ r,
                float* __restrict__ z, float* __restrict__ p, double* __restrict__ part) {
  __shared__ double sh[32];
  const double inv = 1.0 / sc[SC_S];
  const float pscale = (float)(sc[SC_SOLD] * inv);
  double rz = 0.0, rr = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float ri = (float)(r64[i] * inv);
    const float zi = ri / (float)diag[i];
    r[i] = ri; z[i] = zi;
    p[i] = reset_p ? zi : p[i] * pscale;
    rz = fma((double)ri, (double)zi, rz);
    rr = fma((double)ri, (double)ri, rr);
  }
  rz = block_sum(rz, sh);
  rr = block_sum(rr, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = rz;
    part[gridDim.x + blockIdx.x] = rr;
  }
}

// scalars of the recurrence after an anchor; bb and tol2 are in the scaled units
__global__ void k_mx_anchor_final(const double* __restrict__ part, int nb, double* __restrict__ sc,
                                  const double* __restrict__ bbp, double rtol) {
  __shared__ double sh[32];
  double v[2];
  for (int q = 0; q < 2; ++q) {
    double t = 0.0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) t += part[q * nb + b];
    v[q] = block_sum(t, sh);
  }
  if (threadIdx.x == 0) {
    const double s = sc[SC_S];
    sc[SC_RZ] = v[0];
    sc[SC_RR] = v[1];
    sc[SC_BB] = *bbp / (s * s);
    sc[SC_TOL2] = rtol * rtol;
    sc[SC_CONV] = -1.0;
  }
}

}  // namespace hm

using namespace hm;

namespace {
inline cudaStream_t S_(void* s) { return reinterpret_cast<cudaStream_t>(s); }
inline int grid1(int64_t n, int block) { return (int)((n + block - 1) / block); }
inline int spmv_blocks(int64_t nrow, int per_sm) {
  return (int)std::min<int64_t>((nrow + kSpmvRows - 1) / kSpmvRows, 148 * per_sm);
}
inline int ok_or_cuda() { return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA; }
}  // namespace

extern "C" int hm_csr_spmv(int64_t nrow, const int32_t* indptr, const int32_t* indices,
                           const double* vals, const double* x, double* y, double alpha,
                           double beta, void* stream) {
  if (nrow < 0 || (nrow > 0 && (!indptr || !indices || !vals || !x || !y))) return HM_ERR_ARG;
  if (nrow == 0) return HM_OK;
  k_spmv<8, false, false, 8><<<spmv_blocks(nrow, kSpmvBlocks), 256, 0, S_(stream)>>>(nrow, indptr, indices, nullptr, vals, x, y, alpha, beta, nullptr, nullptr, nullptr);
  return ok_or_cuda();
}

extern "C" int hm_csr_spmv_t(int64_t nrow, const int32_t* indptr, const int32_t* indices,
                             const int32_t* tpos, const double* vals, const double* x, double* y,
                             double alpha, double beta, void* stream) {
  if (nrow < 0 || (nrow > 0 && (!indptr || !indices || !tpos || !vals || !x || !y))) return HM_ERR_ARG;
  if (nrow == 0) return HM_OK;
  k_spmv<8, true, false, 4><<<grid1(nrow, kSpmvRows), 256, 0, S_(stream)>>>(nrow, indptr, indices, tpos, vals, x, y, alpha, beta, nullptr, nullptr, nullptr);
  return ok_or_cuda();
}

extern "C" int hm_csr_diag(int64_t nrow, const int32_t* indptr, const double* vals, double* diag,
                           void* stream) {
  if (nrow < 0 || (nrow > 0 && (!indptr || !vals || !diag))) return HM_ERR_ARG;
  if (nrow == 0) return HM_OK;
  k_csr_diag<<<grid1(nrow, 256), 256, 0, S_(stream)>>>(nrow, indptr, vals, diag);
  return ok_or_cuda();
}

extern "C" int64_t hm_dot_workspace_bytes(int64_t n) {
  (void)n;
  return (int64_t)kReduceBlocks * (int64_t)sizeof(double);
}

extern "C" int hm_dot(int64_t n, const double* x, const double* y, double* out, void* work,
                      void* stream) {
  if (n < 0 || !out || !work || (n > 0 && (!x || !y))) return HM_ERR_ARG;
  double* part = static_cast<double*>(work);
  k_dot_partial<<<reduce_blocks(n), kReduceThreads, 0, S_(stream)>>>(n, x, y, part);
  k_reduce_final<<<1, 1024, 0, S_(stream)>>>(part, reduce_blocks(n), 1, out);
  return ok_or_cuda();
}

// slots for the partial sums of p.q: one per block of the operator (at most n, or
// kReduceBlocks of the CSR product)
inline int64_t pq_slots(int64_t n) { return n > kReduceBlocks ? n : (int64_t)kReduceBlocks; }

extern "C" int64_t hm_pcg_workspace_bytes(int64_t n) {
  // r, z, p, q, the partial sums of p.q, scalars, partials
  return (int64_t)sizeof(double) * (4 * n + pq_slots(n) + SC_N + 3 * (int64_t)kReduceBlocks + 8);
}

int hm_pcg_operator(int64_t n, const int32_t* indptr, const int32_t* indices, const double* vals,
                    const hm::Lattice* L, const void* quad, int precision, const uint8_t* ess,
                    const double* x, double* y, void* stream, double* fail);

namespace {

// The operator of one PCG: y = A x; with part (and counter) a CG step's product, whose
// last block also takes the step's alpha from the partial sums of x.y.  sc[SC_FAIL] is set
// where the matrix-free operator gives up a wait.
struct PcgOp {
  int64_t n;
  const int32_t* indptr;
  const int32_t* indices;
  const double* vals;
  const hm::Lattice* L;
  void* jac;
  int precision;
  const uint8_t* ess;
};

int op_apply(const PcgOp& o, const double* x, double* y, void* stream, double* sc, double* part = nullptr,
             unsigned* counter = nullptr) {
  if (part == nullptr)
    return hm_pcg_operator(o.n, o.indptr, o.indices, o.vals, o.L, o.jac, o.L ? o.precision : HM_FP64, o.ess, x, y,
                           stream, sc + SC_FAIL);
  if (o.L != nullptr) return hm_launch_apply_A_dot(*o.L, o.jac, o.precision, o.ess, x, y, part, stream, sc, counter);
  k_spmv<8, false, true, 8><<<spmv_blocks(o.n, kSpmvDotBlocks), 256, 0, S_(stream)>>>(o.n, o.indptr, o.indices, nullptr, o.vals, x, y,
                                                                     1.0, 0.0, part, sc, counter);
  return ok_or_cuda();
}

int op_apply(const PcgOp& o, const float* x, float* y, void* stream, double* sc, double* part = nullptr,
             unsigned* counter = nullptr) {
  return hm_launch_apply_A32_dot(*o.L, o.jac, o.ess, x, y, part, stream, sc, counter);
}

// the two counters of a solve (pcg_batch), zero between uses
inline unsigned* solve_counters(double* sc) { return reinterpret_cast<unsigned*>(sc + SC_CNT); }
// at a solve's start: the counters, and no pass has failed
int reset_counters(double* sc, cudaStream_t s) {
  static_assert(SC_CNT == SC_FAIL + 1 && sizeof(double) == 2 * sizeof(unsigned), "one fill");
  return cudaMemsetAsync(sc + SC_FAIL, 0, 2 * sizeof(double), s) == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

// `count` PCG iterations (operator with p.q and alpha, update with r.z and r.r, beta,
// direction); nothing in it synchronises with the host
// cnt: two counters (zero between uses) for the reductions the producing kernels finish
template <typename T>
int pcg_batch(const PcgOp& o, const double* diag, T* x, T* r, T* z, T* p, T* q, double* pq_part,
              double* sc, double* part, unsigned* cnt, int count, cudaStream_t s) {
  for (int j = 0; j < count; ++j) {
    const int rc = op_apply(o, p, q, (void*)s, sc, pq_part, cnt);
    if (rc) return rc;
    k_pcg_update<T><<<reduce_blocks(o.n), kReduceThreads, 0, s>>>(o.n, sc, x, r, z, p, q, diag, part,
                                                               cnt + 1);
    k_pcg_pupdate<T><<<reduce_blocks(o.n), kReduceThreads, 0, s>>>(o.n, sc, z, p);
  }
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

}  // namespace

// A full batch of iterations captured once as a CUDA graph and replayed (a solve plan
// owns one per precision); partial batches, and streams that cannot be captured (the
// legacy default stream), launch directly.
struct HmBatchGraph {
  cudaGraphExec_t exec = nullptr;
  ~HmBatchGraph() {
    if (exec) cudaGraphExecDestroy(exec);
  }
};

namespace {

template <typename F>
int run_batch(HmBatchGraph* g, bool full, cudaStream_t s, F&& launch) {
  if (g == nullptr || s == nullptr || !full) return launch();
  if (g->exec == nullptr) {
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return HM_ERR_CUDA;
    const int rc = launch();
    const cudaError_t e = cudaStreamEndCapture(s, &graph);
    if (rc != HM_OK || e != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      (void)cudaGetLastError();
      return rc != HM_OK ? rc : HM_ERR_CUDA;
    }
    const cudaError_t ei = cudaGraphInstantiate(&g->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) {
      g->exec = nullptr;
      return HM_ERR_CUDA;
    }
  }
  return cudaGraphLaunch(g->exec, s) == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

// Jacobi-PCG on vectors of type T from initial guess x; work holds r, z, p, q (T), the
// p.q partials (n doubles), the scalars and the partials.  Returns HM_OK / HM_ERR_NOCONV.
template <typename T>
int pcg_run(const PcgOp& o, const double* diag, const T* b, T* x, double rtol, int maxiter,
            int check_every, double* wd, T* wt, int* iterations, double* relres, void* stream,
            HmBatchGraph* graph = nullptr) {
  const int64_t n = o.n;
  cudaStream_t s = S_(stream);
  T* r = wt;
  T* z = wt + n;
  T* p = wt + 2 * n;
  T* q = wt + 3 * n;
  double* pq_part = wd;
  double* sc = wd + pq_slots(n);
  double* part = sc + SC_N;
  unsigned* cnt = solve_counters(sc);
  if (check_every <= 0) check_every = 1;
  if (reset_counters(sc, s) != HM_OK) return HM_ERR_CUDA;
  int rc;
  // x = b on the Dirichlet nodes: every residual and direction is then zero there, which
  // the lattice operator's direction products rely on
  if constexpr (std::is_same<T, double>::value)
    if (o.L && (rc = hm_launch_ess_take_b(*o.L, o.ess, b, x, stream))) return rc;
  rc = op_apply(o, x, q, stream, sc);
  if (rc) return rc;
  k_pcg_init<T><<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, b, q, diag, r, z, p, part);
  k_pcg_init_final<<<1, 1024, 0, s>>>(part, reduce_blocks(n), sc, rtol);
  double host[SC_N];
  int it = 0;
  for (;;) {
    if (cudaMemcpyAsync(host, sc, sizeof(host), cudaMemcpyDeviceToHost, s) != cudaSuccess) return HM_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess || host[SC_FAIL] != 0.0) return HM_ERR_CUDA;
    if (host[SC_CONV] >= 0.0 || it >= maxiter) break;
    const int count = it + check_every < maxiter ? check_every : maxiter - it;
    rc = run_batch(graph, count == check_every, s, [&] {
      return pcg_batch<T>(o, diag, x, r, z, p, q, pq_part, sc, part, cnt, count, s);
    });
    if (rc) return rc;
    it += count;
  }
  const bool conv = host[SC_CONV] >= 0.0;
  if (iterations) *iterations = conv ? (int)host[SC_CONV] : it;
  if (relres) *relres = host[SC_BB] > 0.0 ? std::sqrt(host[SC_RR] / host[SC_BB]) : 0.0;
  return conv ? HM_OK : HM_ERR_NOCONV;
}

}  // namespace

extern "C" int hm_pcg_impl(int64_t n, const int32_t* indptr, const int32_t* indices,
                           const double* vals, const hm::Lattice* L, const void* quad,
                           int precision, const uint8_t* ess, const double* diag, const double* b,
                           double* x, double rtol, int maxiter, int check_every, void* work,
                           int* iterations, double* relres, void* stream) {
  if (n <= 0 || !diag || !b || !x || !work || maxiter < 0) return HM_ERR_ARG;
  PcgOp o{n, indptr, indices, vals, L, const_cast<void*>(quad), precision, ess};
  double* w = static_cast<double*>(work);
  return pcg_run<double>(o, diag, b, x, rtol, maxiter, check_every, w + 4 * n, w, iterations,
                         relres, stream);
}

// the V-cycle is symmetric only to rounding (FP32): its CG takes the flexible step
bool hm_mg_flexible(const hm_mg* mg);
const double* hm_mg_level0_diag(const hm_mg* mg);
void* hm_mg_jac(const hm_mg* mg);
const uint8_t* hm_mg_ess(const hm_mg* mg);
const hm::Lattice* hm_mg_lattice(const hm_mg* mg);

namespace {
// PCG preconditioned by a multigrid V-cycle (the operator and diagonal are the MG's
// level 0); work as for hm_pcg.  x is the initial guess.
int pcg_mg_run(hm_mg* mg, const double* b, double* x, double rtol, int maxiter, int check_every,
               void* work, int* iterations, double* relres, void* stream, HmBatchGraph* graph) {
  const hm::Lattice* L = hm_mg_lattice(mg);
  if (!L || !hm_mg_jac(mg)) return HM_ERR_ARG;
  const int64_t n = L->ndof;
  cudaStream_t s = S_(stream);
  PcgOp o{n, nullptr, nullptr, nullptr, L, hm_mg_jac(mg), HM_FP64, hm_mg_ess(mg)};
  double* w = static_cast<double*>(work);
  double* r = w;
  double* z = w + n;
  double* p = w + 2 * n;
  double* q = w + 3 * n;
  double* pq_part = w + 4 * n;
  double* sc = pq_part + pq_slots(n);
  double* part = sc + SC_N;
  unsigned* cnt = solve_counters(sc);
  if (check_every <= 0) check_every = 1;
  if (reset_counters(sc, s) != HM_OK) return HM_ERR_CUDA;
  int rc = hm_launch_ess_take_b(*L, o.ess, b, x, stream);   // as in pcg_run
  if (rc) return rc;
  rc = op_apply(o, x, q, stream, sc);
  if (rc) return rc;
  const HmFirstDir fd = hm_mg_first_dir(mg);
  k_pcg_mg_init<<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, b, q, r, part, fd);
  if ((rc = hm_mg_vcycle(mg, r, z, stream, sc + SC_FAIL))) return rc;
  k_dot_partial_t<double><<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, r, z, part);
  k_pcg_init_final<<<1, 1024, 0, s>>>(part, reduce_blocks(n), sc, rtol);
  if (cudaMemcpyAsync(p, z, sizeof(double) * n, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return HM_ERR_CUDA;
  double host[SC_N];
  int it = 0;
  const int flex = hm_mg_flexible(mg) ? 1 : 0;
  // with the FP32 cycle: r.r at each check; the solve stops (HM_ERR_NOCONV) once, past
  // iteration 24, twelve iterations no longer halve the residual -- the cycle's rounding,
  // relative to the smooth part of its correction, then swamps the rest (high contrast)
  std::vector<double> hist;
  const int back = (12 + check_every - 1) / check_every;
  bool stalled = false;
  for (;;) {
    if (cudaMemcpyAsync(host, sc, sizeof(host), cudaMemcpyDeviceToHost, s) != cudaSuccess) return HM_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess || host[SC_FAIL] != 0.0) return HM_ERR_CUDA;
    if (host[SC_CONV] >= 0.0 || it >= maxiter) break;
    if (flex) {
      hist.push_back(host[SC_RR]);
      if (it >= 24 && (int)hist.size() > back &&
          host[SC_RR] > 0.25 * hist[hist.size() - 1 - back]) {
        stalled = true;
        break;
      }
    }
    const int count = it + check_every < maxiter ? check_every : maxiter - it;
    rc = run_batch(graph, count == check_every, s, [&]() -> int {
      for (int j = 0; j < count; ++j) {
        int e = op_apply(o, p, q, (void*)s, sc, pq_part, cnt);
        if (e) return e;
        k_pcg_update_rr<<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, sc, x, r, p, q, part, fd,
                                                                 flex ? z : nullptr);
        // the cycle's last operator pass takes r.z and the step's beta where it can
        HmBeta be{pq_part, part + reduce_blocks(n), (unsigned)reduce_blocks(n), flex, sc, cnt + 1, 0};
        if ((e = hm_mg_vcycle(mg, r, z, (void*)s, sc + SC_FAIL, &be))) return e;
        if (!be.done && (e = hm_launch_beta(*L, r, z, be, (void*)s))) return e;
        k_pcg_pupdate<double><<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, sc, z, p);
      }
      return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
    });
    if (rc) return rc;
    it += count;
  }
  const bool conv = !stalled && host[SC_CONV] >= 0.0;
  if (iterations) *iterations = conv ? (int)host[SC_CONV] : it;
  if (relres) *relres = host[SC_BB] > 0.0 ? std::sqrt(host[SC_RR] / host[SC_BB]) : 0.0;
  return conv ? HM_OK : HM_ERR_NOCONV;
}
}  // namespace

extern "C" int hm_pcg_mg(hm_mg* mg, const double* b, double* x, double rtol, int maxiter,
                         int check_every, void* work, int* iterations, double* relres,
                         void* stream) {
  if (!mg || !b || !x || !work || maxiter < 0) return HM_ERR_ARG;
  return pcg_mg_run(mg, b, x, rtol, maxiter, check_every, work, iterations, relres, stream,
                    nullptr);
}

extern "C" int64_t hm_pcg_mixed_workspace_bytes(int64_t n) {
  // FP64: r, t, the p.q partials (at most one per node), scalars, partials, b.b;
  // FP32: x, r, z, p, q of the single-precision recurrence
  return (int64_t)sizeof(double) * (4 * n + pq_slots(n) + SC_N + 3 * (int64_t)kReduceBlocks + 8) +
         (int64_t)sizeof(float) * (5 * n + 16);
}

// Conjugate gradients with reliable updates (Sleijpen & van der Vorst, 1996): the
// recurrence runs in FP32 (vectors and the FP32 matrix-free operator, sums in FP64) on
// a system scaled by the residual norm s; when its residual has fallen by `delta` since
// the last anchor, or it claims convergence, the correction is added to the FP64 x,
// the true residual b - A64 x replaces the recurrence's (rescaled; the search direction
// is kept), and the true residual decides convergence.  Goal and stall test follow the
// reference's refined solves (modeling/PDEVariationalProblem.py:1236-1237, :1299): a
// residual that no longer halves between anchors is at its rounding floor; it counts as
// converged within 10 rtol.
namespace {
int pcg_mixed_run(const hm::Lattice* L, void* jac64, void* jac32, const uint8_t* ess,
                  const double* diag, const double* b, double* x, double rtol, double delta,
                  int max_updates, int maxiter, int check_every, void* work, int* iterations,
                  int* updates, double* relres, void* stream, HmBatchGraph* graph) {
  if (!L || !jac64 || !jac32 || !diag || !b || !x || !work || max_updates <= 0 || maxiter < 0 ||
      !(delta > 0.0 && delta < 1.0) || !(rtol >= 0.0))
    return HM_ERR_ARG;
  const int64_t n = L->ndof;
  cudaStream_t s = S_(stream);
  double* w = static_cast<double*>(work);
  double* r64 = w;
  double* t64 = w + n;
  double* pq_part = w + 4 * n;     // (w + 2n .. 4n: the FP64 finish's z and p)
  double* sc = pq_part + pq_slots(n);
  double* part = sc + SC_N;
  double* bbp = part + 3 * kReduceBlocks;
  unsigned* cnt = solve_counters(sc);
  float* f32 = reinterpret_cast<float*>(bbp + 8);
  float* x32 = f32;
  float* r32 = f32 + n;
  float* z32 = f32 + 2 * n;
  float* p32 = f32 + 3 * n;
  float* q32 = f32 + 4 * n;
  PcgOp o32{n, nullptr, nullptr, nullptr, L, jac32, HM_FP32, ess};
  PcgOp o64{n, nullptr, nullptr, nullptr, L, jac64, HM_FP64, ess};
  if (check_every <= 0) check_every = 1;
  double h[SC_N];
  auto read = [&]() -> int {
    if (cudaMemcpyAsync(h, sc, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess) return HM_ERR_CUDA;
    return cudaStreamSynchronize(s) == cudaSuccess && h[SC_FAIL] == 0.0 ? HM_OK : HM_ERR_CUDA;
  };
  // the anchor: [x += s x32; t = A64 x]; r = b - t; new scale; FP32 r, z, p from r (p
  // restarted as z on the first anchor and on a restart)
  auto anchor = [&](bool first, bool restart) -> int {
    if (!first) {
      k_mx_accum<<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, sc, x32, x);
      const int rc = op_apply(o64, x, t64, stream, sc);
      if (rc) return rc;
    }
    // first: x is b on the Dirichlet nodes and 0 elsewhere, so r = b off them, 0 on them
    k_residual64<<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, b, first ? nullptr : t64,
                                                          first ? ess : nullptr, r64, part);
    k_mx_scale<<<1, 1024, 0, s>>>(part, reduce_blocks(n), sc);
    if (first && cudaMemcpyAsync(bbp, sc + SC_TRUE, sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      return HM_ERR_CUDA;
    k_mx_anchor<<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, r64, diag, sc, (first || restart) ? 1 : 0,
                                                         r32, z32, p32, part);
    k_mx_anchor_final<<<1, 1024, 0, s>>>(part, reduce_blocks(n), sc, bbp, rtol);
    if (cudaGetLastError() != cudaSuccess) return HM_ERR_CUDA;
    return read();
  };
  if (cudaMemsetAsync(sc, 0, sizeof(double) * SC_N, s) != cudaSuccess ||
      cudaMemsetAsync(x, 0, sizeof(double) * n, s) != cudaSuccess ||
      cudaMemsetAsync(x32, 0, sizeof(float) * n, s) != cudaSuccess)
    return HM_ERR_CUDA;
  int rc = hm_launch_ess_take_b(*L, ess, b, x, stream);
  if (rc) return rc;
  rc = anchor(true, true);
  if (rc) return rc;
  const double bb = h[SC_TRUE];
  const double tol2 = rtol * rtol * bb, goal2 = 100.0 * tol2;
  double tr = bb, prev = bb;
  int it = 0, nup = 0, stalls = 0, last_anchor = 0;
  bool conv = tr <= tol2;
  while (!conv) {
    const int count = it + check_every < maxiter ? check_every : maxiter - it;
    rc = run_batch(graph, count == check_every, s, [&] {
      return pcg_batch<float>(o32, diag, x32, r32, z32, p32, q32, pq_part, sc, part, cnt, count, s);
    });
    if (rc) return rc;
    it += count;
    if ((rc = read())) return rc;
    const bool claim = h[SC_CONV] >= 0.0;
    // a recurrence that has grown above its anchor's residual, or has not fallen by
    // delta in 2000 iterations, has lost its way in single precision: restart it
    const bool lost = !(h[SC_RR] <= 1.0) || it - last_anchor > 2000;
    if (!claim && !lost && h[SC_RR] > delta * delta && it < maxiter) continue;
    if ((rc = anchor(false, lost))) return rc;
    last_anchor = it;
    ++nup;
    tr = h[SC_TRUE];
    if (tr <= tol2) { conv = true; break; }
    const bool stalled = tr > 0.25 * prev;
    stalls = stalled ? stalls + 1 : 0;
    prev = tr;
    if ((stalled && claim) || stalls >= 2 || it >= maxiter || nup >= max_updates) {
      conv = tr <= goal2;
      break;
    }
  }
  if (!conv && it < maxiter) {
    // single precision cannot carry this solve (its residual stalls above the goal, or
    // the anchors run out): finish it in FP64 from the current x, as the reference's
    // refined solves do (_solve_in_double, modeling/PDEVariationalProblem.py:1329-1360)
    int its64 = 0;
    double rr64 = 0.0;
    const int rc64 = pcg_run<double>(o64, diag, b, x, rtol, maxiter - it, check_every, pq_part,
                                     w, &its64, &rr64, stream);
    if (rc64 != HM_OK && rc64 != HM_ERR_NOCONV) return rc64;
    if (iterations) *iterations = it + its64;
    if (updates) *updates = nup;
    if (relres) *relres = rr64;
    return rc64;
  }
  if (iterations) *iterations = it;
  if (updates) *updates = nup;
  if (relres) *relres = bb > 0.0 ? std::sqrt(tr / bb) : 0.0;
  return conv ? HM_OK : HM_ERR_NOCONV;
}
}  // namespace

extern "C" int hm_pcg_mixed_impl(const hm::Lattice* L, void* jac64, void* jac32, const uint8_t* ess,
                                 const double* diag, const double* b, double* x, double rtol,
                                 double delta, int max_updates, int maxiter, int check_every,
                                 void* work, int* iterations, int* updates, double* relres,
                                 void* stream) {
  return pcg_mixed_run(L, jac64, jac32, ess, diag, b, x, rtol, delta, max_updates, maxiter,
                       check_every, work, iterations, updates, relres, stream, nullptr);
}

// ------------------------------------------------------------------ solve plans
struct hm_pcg_plan {
  hm::Lattice L;
  void* jac64;
  void* jac32;          // NULL: an FP64 solve
  const uint8_t* ess;
  const double* diag;
  double* b;
  double* x;
  void* work;
  int check_every;
  hm_mg* mg;            // non-NULL: MG-preconditioned FP64 solves
  HmBatchGraph graph;
};

extern "C" int hm_pcg_plan_create(const hm_lattice* h, void* jac64, void* jac32,
                                  const uint8_t* ess, const double* diag, double* b, double* x,
                                  void* work, int check_every, hm_pcg_plan** plan) {
  const hm::Lattice* L = hm_lattice_geometry(h);
  if (!L || !jac64 || !diag || !b || !x || !work || !plan || check_every <= 0) return HM_ERR_ARG;
  hm_pcg_plan* p = new (std::nothrow) hm_pcg_plan();
  if (!p) return HM_ERR_NOMEM;
  p->L = *L;
  p->jac64 = jac64;
  p->jac32 = jac32;
  p->ess = ess;
  p->diag = diag;
  p->b = b;
  p->x = x;
  p->work = work;
  p->check_every = check_every;
  p->mg = nullptr;
  *plan = p;
  return HM_OK;
}

int hm_plan_buffers(const hm_pcg_plan* p, double** b, double** x) {
  if (!p || !b || !x) return HM_ERR_ARG;
  *b = p->b;
  *x = p->x;
  return HM_OK;
}

extern "C" int hm_pcg_plan_set_mg(hm_pcg_plan* p, hm_mg* mg) {
  if (!p || (mg && p->jac32 != nullptr)) return HM_ERR_ARG;
  if (p->graph.exec) {
    cudaGraphExecDestroy(p->graph.exec);
    p->graph.exec = nullptr;
  }
  p->mg = mg;
  return HM_OK;
}

extern "C" int hm_pcg_plan_solve(hm_pcg_plan* p, double rtol, double delta, int max_updates,
                                 int maxiter, int* iterations, int* updates, double* relres,
                                 void* stream) {
  if (!p || maxiter < 0) return HM_ERR_ARG;
  if (p->mg != nullptr) {
    if (updates) *updates = 0;
    if (cudaMemsetAsync(p->x, 0, sizeof(double) * p->L.ndof, S_(stream)) != cudaSuccess)
      return HM_ERR_CUDA;
    return pcg_mg_run(p->mg, p->b, p->x, rtol, maxiter, p->check_every, p->work, iterations,
                      relres, stream, &p->graph);
  }
  if (p->jac32 != nullptr)
    return pcg_mixed_run(&p->L, p->jac64, p->jac32, p->ess, p->diag, p->b, p->x, rtol, delta,
                         max_updates, maxiter, p->check_every, p->work, iterations, updates,
                         relres, stream, &p->graph);
  const int64_t n = p->L.ndof;
  cudaStream_t s = S_(stream);
  if (cudaMemsetAsync(p->x, 0, sizeof(double) * n, s) != cudaSuccess) return HM_ERR_CUDA;
  PcgOp o{n, nullptr, nullptr, nullptr, &p->L, p->jac64, HM_FP64, p->ess};
  double* w = static_cast<double*>(p->work);
  if (updates) *updates = 0;
  return pcg_run<double>(o, p->diag, p->b, p->x, rtol, maxiter, p->check_every, w + 4 * n, w,
                         iterations, relres, stream, &p->graph);
}

extern "C" int hm_pcg_plan_destroy(hm_pcg_plan* p) {
  delete p;
  return HM_OK;
}

// ------------------------------------------------------------------- solve groups
// Several FP64 solve plans of one lattice size solved together: every plan's iteration
// batch is one branch of a single CUDA graph (one launch runs the batches of all
// plans, concurrently on the device), and one host synchronisation per batch reads
// every plan's convergence.  Each branch launches exactly the kernels its plan launches
// alone, on its own buffers, and a converged plan's iterate is frozen (its step length
// is zero), so every result is the one the plan gives solved alone, bit for bit.
struct hm_pcg_group {
  std::vector<hm_pcg_plan*> plans;
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> join;
  cudaEvent_t fork = nullptr;
  cudaGraphExec_t exec = nullptr;
  int check_every = 1;
  ~hm_pcg_group() {
    if (exec) cudaGraphExecDestroy(exec);
    for (auto e : join) cudaEventDestroy(e);
    if (fork) cudaEventDestroy(fork);
    for (auto s : side) cudaStreamDestroy(s);
  }
};

namespace {
struct PlanBufs {
  double *r, *z, *p, *q, *pq_part, *sc, *part;
  unsigned* cnt;
};
PlanBufs plan_bufs(const hm_pcg_plan* pl) {
  const int64_t n = pl->L.ndof;
  double* w = static_cast<double*>(pl->work);
  PlanBufs b;
  b.r = w; b.z = w + n; b.p = w + 2 * n; b.q = w + 3 * n;
  b.pq_part = w + 4 * n;
  b.sc = b.pq_part + pq_slots(n);
  b.part = b.sc + SC_N;
  b.cnt = solve_counters(b.sc);
  return b;
}

// a plan's solve up to its first convergence check (x from zero), as its own solve does
int group_init(hm_pcg_plan* pl, double rtol, cudaStream_t s) {
  const int64_t n = pl->L.ndof;
  const PlanBufs B = plan_bufs(pl);
  PcgOp o{n, nullptr, nullptr, nullptr, &pl->L, pl->jac64, HM_FP64, pl->ess};
  if (cudaMemsetAsync(pl->x, 0, sizeof(double) * n, s) != cudaSuccess || reset_counters(B.sc, s) != HM_OK)
    return HM_ERR_CUDA;
  int rc = hm_launch_ess_take_b(pl->L, o.ess, pl->b, pl->x, (void*)s);
  if (rc) return rc;
  if ((rc = op_apply(o, pl->x, B.q, (void*)s, B.sc))) return rc;
  if (pl->mg != nullptr) {
    k_pcg_mg_init<<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, pl->b, B.q, B.r, B.part,
                                                           hm_mg_first_dir(pl->mg));
    if ((rc = hm_mg_vcycle(pl->mg, B.r, B.z, (void*)s, B.sc + SC_FAIL))) return rc;
    k_dot_partial_t<double><<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, B.r, B.z, B.part);
    k_pcg_init_final<<<1, 1024, 0, s>>>(B.part, reduce_blocks(n), B.sc, rtol);
    if (cudaMemcpyAsync(B.p, B.z, sizeof(double) * n, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      return HM_ERR_CUDA;
  } else {
    k_pcg_init<double><<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, pl->b, B.q, pl->diag, B.r, B.z,
                                                               B.p, B.part);
    k_pcg_init_final<<<1, 1024, 0, s>>>(B.part, reduce_blocks(n), B.sc, rtol);
  }
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

// `count` iterations of a plan, the same launches as its own solve's batches
int group_batch(hm_pcg_plan* pl, int count, cudaStream_t s) {
  const int64_t n = pl->L.ndof;
  const PlanBufs B = plan_bufs(pl);
  PcgOp o{n, nullptr, nullptr, nullptr, &pl->L, pl->jac64, HM_FP64, pl->ess};
  if (pl->mg == nullptr)
    return pcg_batch<double>(o, pl->diag, pl->x, B.r, B.z, B.p, B.q, B.pq_part, B.sc, B.part,
                             B.cnt, count, s);
  for (int j = 0; j < count; ++j) {
    int e = op_apply(o, B.p, B.q, (void*)s, B.sc, B.pq_part, B.cnt);
    if (e) return e;
    const int flex = hm_mg_flexible(pl->mg) ? 1 : 0;
    k_pcg_update_rr<<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, B.sc, pl->x, B.r, B.p, B.q, B.part,
                                                             hm_mg_first_dir(pl->mg),
                                                             flex ? B.z : nullptr);
    HmBeta be{B.pq_part, B.part + reduce_blocks(n), (unsigned)reduce_blocks(n), flex, B.sc, B.cnt + 1, 0};
    if ((e = hm_mg_vcycle(pl->mg, B.r, B.z, (void*)s, B.sc + SC_FAIL, &be))) return e;
    if (!be.done && (e = hm_launch_beta(pl->L, B.r, B.z, be, (void*)s))) return e;
    k_pcg_pupdate<double><<<reduce_blocks(n), kReduceThreads, 0, s>>>(n, B.sc, B.z, B.p);
  }
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}
}  // namespace

extern "C" int hm_pcg_group_create(hm_pcg_plan** plans, int count, hm_pcg_group** out) {
  if (!plans || count < 1 || count > 64 || !out) return HM_ERR_ARG;
  for (int i = 0; i < count; ++i) {
    if (!plans[i] || plans[i]->jac32 != nullptr) return HM_ERR_ARG;   // FP64 plans only
    if (plans[i]->check_every != plans[0]->check_every) return HM_ERR_ARG;
    for (int j = 0; j < i; ++j)
      if (plans[j] == plans[i]) return HM_ERR_ARG;
  }
  hm_pcg_group* g = new (std::nothrow) hm_pcg_group();
  if (!g) return HM_ERR_NOMEM;
  g->plans.assign(plans, plans + count);
  g->check_every = plans[0]->check_every;
  if (cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming) != cudaSuccess) {
    delete g;
    return HM_ERR_CUDA;
  }
  for (int i = 0; i < count; ++i) {
    cudaStream_t st = nullptr;
    cudaEvent_t ev = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
      delete g;
      return HM_ERR_CUDA;
    }
    g->side.push_back(st);
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
      delete g;
      return HM_ERR_CUDA;
    }
    g->join.push_back(ev);
  }
  *out = g;
  return HM_OK;
}

extern "C" int hm_pcg_group_destroy(hm_pcg_group* g) {
  delete g;
  return HM_OK;
}

extern "C" int hm_pcg_group_solve(hm_pcg_group* g, double rtol, int maxiter, int* iterations,
                                  double* relres, void* stream) {
  if (!g || maxiter < 0 || !(rtol >= 0.0)) return HM_ERR_ARG;
  cudaStream_t s = S_(stream);
  const int k = (int)g->plans.size();
  int rc;
  for (int i = 0; i < k; ++i)
    if ((rc = group_init(g->plans[i], rtol, s))) return rc;
  std::vector<double> host((size_t)k * SC_N);
  int it = 0;
  bool all = false;
  for (;;) {
    for (int i = 0; i < k; ++i)
      if (cudaMemcpyAsync(&host[(size_t)i * SC_N], plan_bufs(g->plans[i]).sc, SC_N * sizeof(double),
                          cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return HM_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return HM_ERR_CUDA;
    for (int i = 0; i < k; ++i)
      if (host[(size_t)i * SC_N + SC_FAIL] != 0.0) return HM_ERR_CUDA;
    all = true;
    for (int i = 0; i < k; ++i) all = all && host[(size_t)i * SC_N + SC_CONV] >= 0.0;
    if (all || it >= maxiter) break;
    const int count = it + g->check_every < maxiter ? g->check_every : maxiter - it;
    if (s == nullptr || count != g->check_every) {
      for (int i = 0; i < k; ++i)
        if ((rc = group_batch(g->plans[i], count, s))) return rc;
    } else {
      if (g->exec == nullptr) {
        cudaGraph_t graph = nullptr;
        if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return HM_ERR_CUDA;
        int crc = cudaEventRecord(g->fork, s) == cudaSuccess ? HM_OK : HM_ERR_CUDA;
        for (int i = 0; i < k && crc == HM_OK; ++i) {
          if (cudaStreamWaitEvent(g->side[i], g->fork, 0) != cudaSuccess) { crc = HM_ERR_CUDA; break; }
          crc = group_batch(g->plans[i], count, g->side[i]);
          if (crc == HM_OK && (cudaEventRecord(g->join[i], g->side[i]) != cudaSuccess ||
                               cudaStreamWaitEvent(s, g->join[i], 0) != cudaSuccess))
            crc = HM_ERR_CUDA;
        }
        const cudaError_t e = cudaStreamEndCapture(s, &graph);
        if (crc != HM_OK || e != cudaSuccess) {
          if (graph) cudaGraphDestroy(graph);
          (void)cudaGetLastError();
          return crc != HM_OK ? crc : HM_ERR_CUDA;
        }
        const cudaError_t ei = cudaGraphInstantiate(&g->exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ei != cudaSuccess) {
          g->exec = nullptr;
          return HM_ERR_CUDA;
        }
      }
      if (cudaGraphLaunch(g->exec, s) != cudaSuccess) return HM_ERR_CUDA;
    }
    it += count;
  }
  for (int i = 0; i < k; ++i) {
    const double* h = &host[(size_t)i * SC_N];
    const bool conv = h[SC_CONV] >= 0.0;
    if (iterations) iterations[i] = conv ? (int)h[SC_CONV] : it;
    if (relres) relres[i] = h[SC_BB] > 0.0 ? std::sqrt(h[SC_RR] / h[SC_BB]) : 0.0;
  }
  return all ? HM_OK : HM_ERR_NOCONV;
}
