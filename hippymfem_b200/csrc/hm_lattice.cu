// Structured-lattice kernels of the Q2 log-conductivity path (sm_100a).
//
//   k_pattern_*     the CSR graph (diagonal first), the entry->slot map and the
//                   transpose map of a Q2 x Q2 block, arithmetically
//   k_quad          pointwise data D, E = D grad u, F = D grad p, W = D grad u.grad p
//   k_extract_D     the matrix-free Jacobian's data (its apply is in hm_apply.cu)
//   k_elem_vectors, the assembled vectors by element results and a gather, for small meshes
//   k_node_gather   and outputs that overlap the fields (the others are in hm_apply.cu)
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
// Layout: quad[e][c][q], c = 0 D, 1-3 E, 4-6 F, 7 W (each element's 216 values contiguous).
// With mhat, D = w|J| e^m mhat: the data of the directional derivative along mhat
// (the second-order products of the assembled vectors, with f = 0).
//
// Nine threads an element and field, each the three points of a line along x: the
// contractions along y and z are taken once for the three, 39 multiply-adds and 9 shared
// loads a field and point where a thread a point takes 93 and 27.  The points' products and
// the stores follow with a thread a point.
// Bound: the stores, 1728 bytes an element (68 us at 64^3 elements at the copy rate), with
// the FP64 pipe close behind (65), in three phases that only other blocks overlap.  64^3
// elements: 342 us with a thread a point, 189 here; 45 x 52 x 39 120 and 67, 32^3 46 and 26,
// 4^3 3.5 and 3.2.  One set of nine threads for the three fields takes 171 at 64^3 but 4.5
// at 4^3 (the longer chain); 16 elements a block 238, six blocks an SM (spills) 237.
constexpr int kQuadElems = 8;
constexpr int kQuadThreads = 27 * kQuadElems;
constexpr int kQuadBlocks = 5;

// The contractions of a field's nodal values x along y and z at a line's (q2, q3): values,
// and with GRAD derivatives along y and along z, at the three nodes along x.
template <bool GRAD, typename real>
__device__ __forceinline__ void quad_line(const real* x, const real (&b2)[3], const real (&d2)[3],
                                          const real (&b3)[3], const real (&d3)[3], real (&bb)[3],
                                          real (&bd)[3], real (&dz)[3]) {
#pragma unroll
  for (int a1 = 0; a1 < 3; ++a1) bb[a1] = bd[a1] = dz[a1] = real(0);
#pragma unroll
  for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
    for (int a1 = 0; a1 < 3; ++a1) {
      real sb = 0, sd = 0;
#pragma unroll
      for (int a2 = 0; a2 < 3; ++a2) {
        const real v = x[a1 + 3 * a2 + 9 * a3];
        sb = fma(b2[a2], v, sb);
        if constexpr (GRAD) sd = fma(d2[a2], v, sd);
      }
      bb[a1] = fma(b3[a3], sb, bb[a1]);
      if constexpr (GRAD) {
        bd[a1] = fma(b3[a3], sd, bd[a1]);
        dz[a1] = fma(d3[a3], sb, dz[a1]);
      }
    }
}

template <typename real, bool MHAT>
__global__ void __launch_bounds__(kQuadThreads, kQuadBlocks)
    k_quad(Lattice L, const double* __restrict__ u,
           const double* __restrict__ m, const double* __restrict__ p, const double* __restrict__ mhat,
           real* __restrict__ quad, uint32_t* __restrict__ status) {
  constexpr int NF = MHAT ? 4 : 3;
  __shared__ real sx[NF][kQuadElems][27];                // m, u, p, mhat
  __shared__ real sg[7][kQuadElems][27];                 // D, grad u, grad p at the points
  __shared__ real sb[3][3], sd[3][3];
  const int tid = threadIdx.x;
  const int64_t e0 = blockIdx.x * (int64_t)kQuadElems;
  const int count = (int)min((int64_t)kQuadElems, L.ne - e0);
  if (tid < 9) {
    sb[tid / 3][tid % 3] = (real)bq(tid / 3, tid % 3);
    sd[tid / 3][tid % 3] = (real)dbq(tid / 3, tid % 3);
  }
  const int pe = tid / 27, a = tid - pe * 27;            // the thread's element as a node or a point
  if (pe < count) {
    const unsigned e = (unsigned)e0 + pe, row = e / (unsigned)L.nx;
    const int ex = (int)(e - row * L.nx), ez = (int)(row / (unsigned)L.ny), ey = (int)(row - (unsigned)ez * L.ny);
    const int64_t node = (2 * ex + a % 3) + (int64_t)L.Nx * ((2 * ey + (a / 3) % 3) + (int64_t)L.Ny * (2 * ez + a / 9));
    sx[0][pe][a] = (real)__ldg(m + node);
    sx[1][pe][a] = (real)__ldg(u + node);
    sx[2][pe][a] = (real)__ldg(p + node);
    if constexpr (MHAT) sx[3][pe][a] = (real)__ldg(mhat + node);
  }
  __syncthreads();
  // a third of the threads a field
  const int f = tid / (9 * kQuadElems), t = tid - f * 9 * kQuadElems;
  const int le = t / 9, line = t - le * 9, q2 = line % 3, q3 = line / 3;
  if (le < count) {
    real b2[3], d2[3], b3[3], d3[3], bb[3], bd[3], dz[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      b2[k] = sb[q2][k]; b3[k] = sb[q3][k];
      d2[k] = sd[q2][k]; d3[k] = sd[q3][k];
    }
    if (f == 0) {
      const double w23 = (q2 == 1 ? wq(1) : wq(0)) * (q3 == 1 ? wq(1) : wq(0)) * L.hx * L.hy * L.hz;
      quad_line<false>(sx[0][le], b2, d2, b3, d3, bb, bd, dz);
      if constexpr (MHAT) quad_line<false>(sx[3][le], b2, d2, b3, d3, dz, bd, d3);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        real v = 0, vh = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          v = fma((real)bq(q, k), bb[k], v);
          if constexpr (MHAT) vh = fma((real)bq(q, k), dz[k], vh);
        }
        real D = (real)(wq(q) * w23) * exp(v);
        if constexpr (MHAT) D *= vh;
        sg[0][le][3 * line + q] = D;
      }
    } else {
      quad_line<true>(sx[f][le], b2, d2, b3, d3, bb, bd, dz);
      // scaled after the contractions: a derivative table's entries cancel exactly on a
      // constant field, divided by the edge they would not
      const real ihx = (real)(1.0 / L.hx), ihy = (real)(1.0 / L.hy), ihz = (real)(1.0 / L.hz);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        real gx = 0, gy = 0, gz = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          gx = fma((real)dbq(q, k), bb[k], gx);
          gy = fma((real)bq(q, k), bd[k], gy);
          gz = fma((real)bq(q, k), dz[k], gz);
        }
        sg[3 * f - 2][le][3 * line + q] = gx * ihx;
        sg[3 * f - 1][le][3 * line + q] = gy * ihy;
        sg[3 * f][le][3 * line + q] = gz * ihz;
      }
    }
  }
  __syncthreads();
  if (pe >= count) return;
  const real D = sg[0][pe][a];
  real* const out = quad + (e0 + pe) * 216 + a;
  real W = 0;
  bool finite = isfinite(D);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const real gu = sg[1 + c][pe][a], gp = sg[4 + c][pe][a];
    const real E = D * gu, F = D * gp;
    W = c == 0 ? gu * gp : W + gu * gp;
    finite = finite && isfinite(E) && isfinite(F);
    out[27 * (1 + c)] = E;
    out[27 * (4 + c)] = F;
  }
  W *= D;
  out[0] = D;
  out[189] = W;
  if (!finite || !isfinite(W)) atomicOr(status, HM_STATUS_NONFINITE);
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

// Diagonal of A(D): sum_g D(g) sum_d (d_d phi_n)^2.  A block owns the nodes of a tile of
// 8 x 4 x 4 elements (and reads one more layer below it): a thread takes one element's 27
// contributions by contractions along x, y and z (567 multiply-adds; 27 x 27 products of
// three factors and three directions node by node), then the nodes sum those of the elements
// that touch them in a fixed order.  Bound: the latency of the loads, 216 of every 1728
// bytes.  64^3 elements: 328 us node by node, 95 here; 45 x 52 x 39 117 and 34; 32^3 48 and
// 13.5; 16^3 10.7 both, 8^3 10.1 and 10.5 (few blocks, each a longer chain; graph replays).
constexpr int kDiagX = 8, kDiagY = 4, kDiagZ = 4;
constexpr int kDiagElems = (kDiagX + 1) * (kDiagY + 1) * (kDiagZ + 1);
// squared derivatives by axis, point and node, divided by the squared edge
struct DiagTab {
  double d2[3][3][3];
};
template <typename real>
__global__ void __launch_bounds__(256, 2)
    k_diag_A(Lattice L, const __grid_constant__ DiagTab tab, const real* __restrict__ quad,
             const uint8_t* __restrict__ ess, double* __restrict__ diag) {
  __shared__ double sD[kDiagElems * 27];
  const int tx = (L.nx + kDiagX - 1) / kDiagX, ty = (L.ny + kDiagY - 1) / kDiagY;
  const int bx = blockIdx.x % tx, by = (blockIdx.x / tx) % ty, bz = blockIdx.x / (tx * ty);
  // the first element of the tile with its lower layer (-1 in the first tile of an axis)
  const int ex0 = bx * kDiagX - 1, ey0 = by * kDiagY - 1, ez0 = bz * kDiagZ - 1;
  // eight loads in flight a thread
  constexpr int kLoads = (kDiagElems * 27 + 255) / 256;
#pragma unroll 1
  for (int r = 0; r < kLoads; r += 8) {
    double v[8];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int t = threadIdx.x + 256 * (r + g), le = t / 27, q = t - le * 27;
      const int ex = ex0 + le % (kDiagX + 1), ey = ey0 + (le / (kDiagX + 1)) % (kDiagY + 1),
                ez = ez0 + le / ((kDiagX + 1) * (kDiagY + 1));
      const bool on = t < kDiagElems * 27 && ex >= 0 && ey >= 0 && ez >= 0 && ex < L.nx && ey < L.ny && ez < L.nz;
      v[g] = on ? (double)__ldg(quad + (ex + (int64_t)L.nx * (ey + (int64_t)L.ny * ez)) * 216 + q) : 0.0;
    }
#pragma unroll
    for (int g = 0; g < 8; ++g)
      if (const int t = threadIdx.x + 256 * (r + g); t < kDiagElems * 27) sD[t] = v[g];
  }
  __syncthreads();
  if (threadIdx.x < kDiagElems) {
    double* const D = sD + threadIdx.x * 27;
    double C[3][3][3];
#pragma unroll
    for (int a = 0; a < 27; ++a) C[a / 9][(a / 3) % 3][a % 3] = 0.0;
#pragma unroll
    for (int q3 = 0; q3 < 3; ++q3) {
      double R[3][3], S[3][3];                 // derivatives along x or y, none
#pragma unroll
      for (int a = 0; a < 9; ++a) R[a / 3][a % 3] = S[a / 3][a % 3] = 0.0;
#pragma unroll
      for (int q2 = 0; q2 < 3; ++q2) {
        double P[3] = {0.0, 0.0, 0.0}, Q[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int q1 = 0; q1 < 3; ++q1) {
          const double v = D[q1 + 3 * q2 + 9 * q3];
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            P[a] = fma(bq(q1, a) * bq(q1, a), v, P[a]);
            Q[a] = fma(tab.d2[0][q1][a], v, Q[a]);
          }
        }
#pragma unroll
        for (int a2 = 0; a2 < 3; ++a2)
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            R[a2][a] = fma(bq(q2, a2) * bq(q2, a2), Q[a], fma(tab.d2[1][q2][a2], P[a], R[a2][a]));
            S[a2][a] = fma(bq(q2, a2) * bq(q2, a2), P[a], S[a2][a]);
          }
      }
#pragma unroll
      for (int a3 = 0; a3 < 3; ++a3)
#pragma unroll
        for (int a = 0; a < 9; ++a)
          C[a3][a / 3][a % 3] = fma(bq(q3, a3) * bq(q3, a3), R[a / 3][a % 3],
                                    fma(tab.d2[2][q3][a3], S[a / 3][a % 3], C[a3][a / 3][a % 3]));
    }
#pragma unroll
    for (int a = 0; a < 27; ++a) D[a] = C[a / 9][(a / 3) % 3][a % 3];
  }
  __syncthreads();
  const int i0 = 2 * (ex0 + 1), j0 = 2 * (ey0 + 1), k0 = 2 * (ez0 + 1);
  // the tile's nodes; the last tile of an axis has the mesh's last node plane as well
  const int ni = i0 + 2 * kDiagX < L.Nx - 1 ? 2 * kDiagX : L.Nx - i0;
  const int nj = j0 + 2 * kDiagY < L.Ny - 1 ? 2 * kDiagY : L.Ny - j0;
  const int nk = k0 + 2 * kDiagZ < L.Nz - 1 ? 2 * kDiagZ : L.Nz - k0;
  for (int t = threadIdx.x; t < ni * nj * nk; t += 256) {
    const int li = t % ni, lj = (t / ni) % nj, lk = t / (ni * nj);
    const int i = i0 + li, j = j0 + lj, k = k0 + lk;
    const int64_t n = i + (int64_t)L.Nx * (j + (int64_t)L.Ny * k);
    // along each axis the element that holds the node as 1, or as 2 and (the next) as 0;
    // elements outside the mesh have zeros
    double acc = 0.0;
    for (int c3 = lk & 1; c3 < 2; ++c3)
      for (int c2 = lj & 1; c2 < 2; ++c2)
        for (int c1 = li & 1; c1 < 2; ++c1) {
          const int e1 = li / 2 + c1, e2 = lj / 2 + c2, e3 = lk / 2 + c3;
          if (e1 > kDiagX || e2 > kDiagY || e3 > kDiagZ) continue;       // past the mesh
          const int a = (li - 2 * (e1 - 1)) + 3 * (lj - 2 * (e2 - 1)) + 9 * (lk - 2 * (e3 - 1));
          acc += sD[(e1 + (kDiagX + 1) * (e2 + (kDiagY + 1) * e3)) * 27 + a];
        }
    diag[n] = ess != nullptr && ess[n] ? 1.0 : acc;
  }
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

namespace {
template <typename real>
int launch_quad(const Lattice& L, const double* u, const double* m, const double* p, const double* mhat,
                real* quad, uint32_t* status, cudaStream_t s) {
  const int blocks = grid1(L.ne, kQuadElems);
  if (mhat) k_quad<real, true><<<blocks, kQuadThreads, 0, s>>>(L, u, m, p, mhat, quad, status);
  else k_quad<real, false><<<blocks, kQuadThreads, 0, s>>>(L, u, m, p, nullptr, quad, status);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}
}  // namespace

int hm_launch_quad(const Lattice& L, const double* u, const double* m, const double* p,
                   int precision, void* quad, uint32_t* status, void* stream, const double* mhat) {
  if (precision == HM_FP32) return launch_quad<float>(L, u, m, p, mhat, static_cast<float*>(quad), status, S_(stream));
  return launch_quad<double>(L, u, m, p, mhat, static_cast<double*>(quad), status, S_(stream));
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
  DiagTab tab;
  const double h[3] = {L.hx, L.hy, L.hz};
  for (int d = 0; d < 3; ++d)
    for (int q = 0; q < 3; ++q)
      for (int a = 0; a < 3; ++a) tab.d2[d][q][a] = dbq(q, a) * dbq(q, a) / (h[d] * h[d]);
  const int blocks = ((L.nx + kDiagX - 1) / kDiagX) * ((L.ny + kDiagY - 1) / kDiagY) * ((L.nz + kDiagZ - 1) / kDiagZ);
  if (precision == HM_FP32)
    k_diag_A<float><<<blocks, 256, 0, S_(stream)>>>(L, tab, (const float*)quad, ess, diag);
  else
    k_diag_A<double><<<blocks, 256, 0, S_(stream)>>>(L, tab, (const double*)quad, ess, diag);
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
// (hm_apply.cu); or the element route below, which reads every field before it writes any
// vector: one pass evaluates the fields at the element's 27 points and contracts the
// element vectors (written as Ye[a][e] into the workspace), the node gather sums them per
// node in a fixed order.
namespace hm {
// Element vectors Ye[a][e] to nodes.  One thread per pair of x-neighbours (2m, 2m+1) of a
// node row (the row's last node, 2n, alone), so that every lane of a warp runs the same
// loop: node 2m takes element m-1 (local a1 = 2) and m (a1 = 0), node 2m+1 element m
// (a1 = 1); consecutive lanes read consecutive elements of each Ye plane.  Per node the
// contributions are summed over (z, y, x) element pairs with the lower element first, a
// fixed order.
__device__ __forceinline__ void axis_elems(int i, int nel, int& e0, int& a0, int& cnt) {
  if (i & 1) { e0 = i >> 1; a0 = 1; cnt = 1; }
  else if (i == 0) { e0 = 0; a0 = 0; cnt = 1; }
  else if ((i >> 1) >= nel) { e0 = (i >> 1) - 1; a0 = 2; cnt = 1; }
  else { e0 = (i >> 1) - 1; a0 = 2; cnt = 2; }   // elements i/2-1 (a=2), i/2 (a=0)
}

__global__ void __launch_bounds__(256)
    k_node_gather(Lattice L, const double* __restrict__ Ye, const uint8_t* __restrict__ zero,
                  double* __restrict__ yout, const uint32_t* __restrict__ skip) {
  if (skip != nullptr && *skip != 0u) return;    // the whole launch stands down
  const unsigned per_row = (unsigned)L.nx + 1u;                  // pairs + the last node
  const unsigned rows = (unsigned)L.Ny * (unsigned)L.Nz;
  const unsigned task = blockIdx.x * blockDim.x + threadIdx.x;
  if (task >= rows * per_row) return;
  const unsigned row = task / per_row;
  const unsigned m = task - row * per_row;
  const unsigned iz = row / (unsigned)L.Ny, iy = row - iz * (unsigned)L.Ny;
  const bool last = m == (unsigned)L.nx;                          // node 2n alone
  const unsigned n0 = row * (unsigned)L.Nx + 2u * m;              // node 2m
  int ey0, ay0, cy, ez0, az0, cz;
  axis_elems((int)iy, L.ny, ey0, ay0, cy);
  axis_elems((int)iz, L.nz, ez0, az0, cz);
  const unsigned ne = (unsigned)L.ne, nx = (unsigned)L.nx;
  // every contribution is loaded before any is added (all twelve loads in flight at
  // once), then summed in the fixed order (z, y element pairs, lower element first)
  double v[4][3];
#pragma unroll
  for (int c3 = 0; c3 < 2; ++c3)
#pragma unroll
    for (int c2 = 0; c2 < 2; ++c2) {
      const int c = 2 * c3 + c2;
      const bool on = c3 < cz && c2 < cy;
      const unsigned a23 = 3u * (unsigned)(c2 ? 0 : ay0) + 9u * (unsigned)(c3 ? 0 : az0);
      const unsigned erow = nx * ((unsigned)(ey0 + c2) + (unsigned)L.ny * (unsigned)(ez0 + c3));
      // node 2m: element m-1 (a1 = 2) then element m (a1 = 0); node 2m+1: element m
      v[c][0] = (on && m > 0) ? Ye[(size_t)(2u + a23) * ne + erow + m - 1u] : 0.0;
      v[c][1] = (on && !last) ? Ye[(size_t)a23 * ne + erow + m] : 0.0;
      v[c][2] = (on && !last) ? Ye[(size_t)(1u + a23) * ne + erow + m] : 0.0;
    }
  double acc0 = 0, acc1 = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if ((c >> 1) < cz && (c & 1) < cy) {
      if (m > 0) acc0 += v[c][0];
      if (!last) {
        acc0 += v[c][1];
        acc1 += v[c][2];
      }
    }
  yout[n0] = zero != nullptr && zero[n0] ? 0.0 : acc0;
  if (!last) yout[n0 + 1] = zero != nullptr && zero[n0 + 1] ? 0.0 : acc1;
}

template <int NV>
struct VecOut { double* ye[3]; };   // element results: ADJOINT, STATE, PARAMETER (NULL: skip)

// Sum factorisation on the element's 3 x 3 x 3 nodes and points: nodes -> points one
// axis at a time (x, y, z), the pointwise data at the 27 points, then points -> nodes
// (z, y, x) for the three element vectors.  One CTA holds 8 elements, a thread per
// (element, index); every stage reads the previous one's arrays in shared memory.
//   evaluation   X: B u, B' u, B p, B' p, B m, B mhat        (index q1 + 3 a2 + 9 a3)
//                Y: u: BB, BB', B'B;  p: the same;  m, mhat: BB  (q1 + 3 q2 + 9 a3)
//                Z: grad u, grad p, m, mhat at the point      (q1 + 3 q2 + 9 q3)
//   integration  Z: E_x B, E_y B, E_z B' + s B | F_x B, F_y B, F_z B' | W B
//                Y: (.) B, (.) B' + (.) B per vector        (q1 + 3 a2 + 9 a3)
//                X: B' (.) + B (.)                          (a1 + 3 a2 + 9 a3)
// with the 1/h of each derivative folded in at its z sums.
__device__ __forceinline__ double b1d(int q, int a) { return bq(q, a); }
__device__ __forceinline__ double d1d(int q, int a) { return dbq(q, a); }

__global__ void __launch_bounds__(216, 4) k_elem_vectors(Lattice L, const double* __restrict__ u,
                                                      const double* __restrict__ m,
                                                      const double* __restrict__ p,
                                                      const double* __restrict__ mhat, double f,
                                                      VecOut<3> o, uint32_t* __restrict__ status,
                                                      const uint32_t* __restrict__ skip) {
  if (skip != nullptr && *skip != 0u) return;    // the whole launch stands down
  // per element: arrays of 27, the element's block padded to 11 (mod 16) doubles, so
  // that the two elements a warp spans fall on different banks
  constexpr int kV = 4 * 27 + 15, kA = 7 * 27 + 14, kB = 8 * 27 + 3;
  __shared__ double sv[8][kV];           // node values u, m, p, mhat
  __shared__ double s1[8][kA];           // evaluation X / integration Z
  __shared__ double s2[8][kB];           // evaluation Y / integration Y
  __shared__ double sp[8][kB];           // E(3), F(3), W, source weight at the points
  const int tid = threadIdx.x, le = tid / 27, i = tid % 27;
  const int c1 = i % 3, c2 = (i / 3) % 3, c3 = i / 9;   // the thread's three indices
  const double ihx = 1.0 / L.hx, ihy = 1.0 / L.hy, ihz = 1.0 / L.hz;
  const double wdet = wq(c1) * wq(c2) * wq(c3) * L.hx * L.hy * L.hz;
  for (int64_t g0 = blockIdx.x * 8LL; g0 < L.ne; g0 += (int64_t)gridDim.x * 8) {
    const int64_t e = g0 + le;
    const bool live = le < 8 && e < L.ne;
    __syncthreads();                      // the previous group's arrays are consumed
    if (live) {
      const int ex = (int)(e % L.nx), ey = (int)((e / L.nx) % L.ny), ez = (int)(e / ((int64_t)L.nx * L.ny));
      const int64_t node = (2 * ex + c1) + (int64_t)L.Nx * ((2 * ey + c2) + (int64_t)L.Ny * (2 * ez + c3));
      // u and p less their value at the element's middle node: only their derivatives
      // are wanted, and the value's rounding over h would be in each
      const int64_t mid = (2 * ex + 1) + (int64_t)L.Nx * ((2 * ey + 1) + (int64_t)L.Ny * (2 * ez + 1));
      sv[le][(0) * 27 + i] = u[node] - u[mid];
      sv[le][(1) * 27 + i] = m[node];
      sv[le][(2) * 27 + i] = p[node] - p[mid];
      sv[le][(3) * 27 + i] = mhat ? mhat[node] : 0.0;
    }
    __syncthreads();
    if (live) {   // X: index (q1 = c1, a2 = c2, a3 = c3), sums over a1
      double r[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int a1 = 0; a1 < 3; ++a1) {
        const int j = a1 + 3 * c2 + 9 * c3;
        const double b = b1d(c1, a1), d = d1d(c1, a1);
        const double vu = sv[le][(0) * 27 + j], vm = sv[le][(1) * 27 + j], vp = sv[le][(2) * 27 + j], vh = sv[le][(3) * 27 + j];
        r[0] = fma(b, vu, r[0]); r[1] = fma(d, vu, r[1]);
        r[2] = fma(b, vp, r[2]); r[3] = fma(d, vp, r[3]);
        r[4] = fma(b, vm, r[4]); r[5] = fma(b, vh, r[5]);
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) s1[le][(k) * 27 + i] = r[k];
    }
    __syncthreads();
    if (live) {   // Y: index (q1 = c1, q2 = c2, a3 = c3), sums over a2
      double r[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int a2 = 0; a2 < 3; ++a2) {
        const int j = c1 + 3 * a2 + 9 * c3;
        const double b = b1d(c2, a2), d = d1d(c2, a2);
        const double x0 = s1[le][(0) * 27 + j], x1 = s1[le][(1) * 27 + j], x2 = s1[le][(2) * 27 + j], x3 = s1[le][(3) * 27 + j];
        r[0] = fma(b, x0, r[0]); r[1] = fma(b, x1, r[1]); r[2] = fma(d, x0, r[2]);
        r[3] = fma(b, x2, r[3]); r[4] = fma(b, x3, r[4]); r[5] = fma(d, x2, r[5]);
        r[6] = fma(b, s1[le][(4) * 27 + j], r[6]); r[7] = fma(b, s1[le][(5) * 27 + j], r[7]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) s2[le][(k) * 27 + i] = r[k];
    }
    __syncthreads();
    if (live) {   // Z: the point (c1, c2, c3), sums over a3; then the pointwise data
      double gu[3] = {0, 0, 0}, gp[3] = {0, 0, 0}, mv = 0.0, mh = 0.0;
#pragma unroll
      for (int a3 = 0; a3 < 3; ++a3) {
        const int j = c1 + 3 * c2 + 9 * a3;
        const double b = b1d(c3, a3), d = d1d(c3, a3);
        gu[0] = fma(b, s2[le][(1) * 27 + j], gu[0]); gu[1] = fma(b, s2[le][(2) * 27 + j], gu[1]);
        gu[2] = fma(d, s2[le][(0) * 27 + j], gu[2]);
        gp[0] = fma(b, s2[le][(4) * 27 + j], gp[0]); gp[1] = fma(b, s2[le][(5) * 27 + j], gp[1]);
        gp[2] = fma(d, s2[le][(3) * 27 + j], gp[2]);
        mv = fma(b, s2[le][(6) * 27 + j], mv); mh = fma(b, s2[le][(7) * 27 + j], mh);
      }
      gu[0] *= ihx; gu[1] *= ihy; gu[2] *= ihz;
      gp[0] *= ihx; gp[1] *= ihy; gp[2] *= ihz;
      double D = wdet * exp(mv);
      if (mhat) D *= mh;
      const double E0 = D * gu[0], E1 = D * gu[1], E2 = D * gu[2];
      const double F0 = D * gp[0], F1 = D * gp[1], F2 = D * gp[2];
      const double W = D * (gu[0] * gp[0] + gu[1] * gp[1] + gu[2] * gp[2]);
      sp[le][(0) * 27 + i] = E0; sp[le][(1) * 27 + i] = E1; sp[le][(2) * 27 + i] = E2;
      sp[le][(3) * 27 + i] = F0; sp[le][(4) * 27 + i] = F1; sp[le][(5) * 27 + i] = F2;
      sp[le][(6) * 27 + i] = W;
      sp[le][(7) * 27 + i] = mhat ? 0.0 : -f * wdet;
      if (!(isfinite(E0) && isfinite(E1) && isfinite(E2) && isfinite(F0) && isfinite(F1) &&
            isfinite(F2) && isfinite(W)))
        atomicOr(status, HM_STATUS_NONFINITE);
    }
    __syncthreads();
    if (live) {   // integration Z: index (q1 = c1, q2 = c2, a3 = c3), sums over q3
      double r[7] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int q3 = 0; q3 < 3; ++q3) {
        const int j = c1 + 3 * c2 + 9 * q3;
        const double b = b1d(q3, c3), d = d1d(q3, c3);
        r[0] = fma(b, sp[le][(0) * 27 + j], r[0]);
        r[1] = fma(b, sp[le][(1) * 27 + j], r[1]);
        r[2] = fma(d * ihz, sp[le][(2) * 27 + j], fma(b, sp[le][(7) * 27 + j], r[2]));
        r[3] = fma(b, sp[le][(3) * 27 + j], r[3]);
        r[4] = fma(b, sp[le][(4) * 27 + j], r[4]);
        r[5] = fma(d, sp[le][(5) * 27 + j], r[5]);
        r[6] = fma(b, sp[le][(6) * 27 + j], r[6]);
      }
      s1[le][(0) * 27 + i] = r[0] * ihx; s1[le][(1) * 27 + i] = r[1] * ihy; s1[le][(2) * 27 + i] = r[2];
      s1[le][(3) * 27 + i] = r[3] * ihx; s1[le][(4) * 27 + i] = r[4] * ihy; s1[le][(5) * 27 + i] = r[5] * ihz;
      s1[le][(6) * 27 + i] = r[6];
    }
    __syncthreads();
    if (live) {   // integration Y: index (q1 = c1, a2 = c2, a3 = c3), sums over q2
      double r[5] = {0, 0, 0, 0, 0};
#pragma unroll
      for (int q2 = 0; q2 < 3; ++q2) {
        const int j = c1 + 3 * q2 + 9 * c3;
        const double b = b1d(q2, c2), d = d1d(q2, c2);
        r[0] = fma(b, s1[le][(0) * 27 + j], r[0]);
        r[1] = fma(d, s1[le][(1) * 27 + j], fma(b, s1[le][(2) * 27 + j], r[1]));
        r[2] = fma(b, s1[le][(3) * 27 + j], r[2]);
        r[3] = fma(d, s1[le][(4) * 27 + j], fma(b, s1[le][(5) * 27 + j], r[3]));
        r[4] = fma(b, s1[le][(6) * 27 + j], r[4]);
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) s2[le][(k) * 27 + i] = r[k];
    }
    __syncthreads();
    if (live) {   // integration X: the node (a1 = c1, a2 = c2, a3 = c3), sums over q1
      double ra = 0.0, rs = 0.0, rp = 0.0;
#pragma unroll
      for (int q1 = 0; q1 < 3; ++q1) {
        const int j = q1 + 3 * c2 + 9 * c3;
        const double b = b1d(q1, c1), d = d1d(q1, c1);
        ra = fma(d, s2[le][(0) * 27 + j], fma(b, s2[le][(1) * 27 + j], ra));
        rs = fma(d, s2[le][(2) * 27 + j], fma(b, s2[le][(3) * 27 + j], rs));
        rp = fma(b, s2[le][(4) * 27 + j], rp);
      }
      if (o.ye[0]) o.ye[0][(int64_t)i * L.ne + e] = ra;
      if (o.ye[1]) o.ye[1][(int64_t)i * L.ne + e] = rs;
      if (o.ye[2]) o.ye[2][(int64_t)i * L.ne + e] = rp;
    }
  }
}

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

namespace {
// the blocks of the gather: one thread per x-pair of every node row
inline int gather_blocks(const Lattice& L) {
  return grid1((int64_t)L.Ny * L.Nz * (L.nx + 1), 256);
}
}  // namespace

// The vectors by the element route: work of 27 ne doubles a vector; outs ADJOINT, STATE,
// PARAMETER (NULL: skip), which may be or overlap any of the fields.  With skip nonzero on
// the device no vector is written.
int hm_launch_elem_vectors(const Lattice& L, const double* u, const double* m, const double* p,
                           const double* mhat, double f, const uint8_t* zero_ess, double* const outs[3],
                           double* work, uint32_t* status, const uint32_t* skip, void* stream) {
  cudaStream_t s = S_(stream);
  VecOut<3> o{};
  int k = 0;
  for (int i = 0; i < 3; ++i)
    if (outs[i]) o.ye[i] = work + (int64_t)(k++) * 27 * L.ne;
  const int64_t groups = (L.ne + 7) / 8;
  k_elem_vectors<<<(int)(groups < 148 * 16 ? groups : 148 * 16), 216, 0, s>>>(L, u, m, p, mhat, f, o, status, skip);
  for (int i = 0; i < 3; ++i)
    if (outs[i])
      k_node_gather<<<gather_blocks(L), 256, 0, s>>>(L, o.ye[i], i != 2 ? zero_ess : nullptr, outs[i], skip);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

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
