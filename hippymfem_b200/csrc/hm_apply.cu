// The matrix-free Jacobian apply y = A(D) x of the Q2 lattice in one pass (sm_100a), with
// the smoothing steps of the multigrid cycle and the inner product of a CG step in its
// epilogue.
//
// A CTA owns a tile of T1 x T2 element columns and marches T3 element layers up z, one
// thread per column (the "cell" (cx, cy, cz) owns the nodes (2cx + {0,1}, 2cy + {0,1},
// 2cz + {0,1}); the cells nx, ny, nz are virtual and own the last node only).  Node planes
// arrive in a ring in shared memory by asynchronous copies, two layers ahead; D of the
// next layer as one TMA box.  Per layer a thread interpolates its
// two new node planes to the 3 x 3 in-plane Gauss points, the three planes to the 27
// points, takes the derivatives *at the Gauss points* (three points carry a quadratic, so
// a 1D derivative is the 3 x 3 matrix (-3 4 -1; -1 0 1; 1 -4 3) / (2 sqrt(0.15))), and goes
// back the same way; every plane enters less its middle node's value, and the three meet
// less the middle plane's, so that the rounding follows the field's variation over the
// element and not its value.  The upper plane's in-plane values, and its sums before they return
// to nodes, stay in the thread for the next layer.  The ten results that other columns'
// nodes need (the element's upper x and y faces on the two lower planes) go through a
// double-buffered exchange, one block barrier a layer, and each thread writes its own 8
// nodes.  A tile recomputes the columns (and the layer) below its first own ones.  Every
// node is summed in one fixed order (the lower layer's sums first, then own column, left,
// front, corner), whatever the tiling: results do not depend on the tile sizes or on how
// a mesh is cut into slabs.
//
// Bound: FP64 arithmetic (~700 operations an element) and its latency.  At 64^3 that is
// 10 us at the full FP64 rate; the 91 MB of traffic take 14 us at the measured copy rate.
// Measured with the product's inner product (CG's A p): 40-42 us at 64^3, 20.7 at 48^3, 13.8
// at 32^3, 8.4 at 16^3, against 80, 37, 16 and 10 us for an element pass (three threads an
// element, element results through memory) and a node gather.  A layer of two CTAs takes
// ~5,000 cycles: ~2,000 the arithmetic (1,400 at the full rate), 1,000 the requests, 950
// the epilogue; 12 warps per SM at 168 registers spill and are slower (81 us).  D as one
// TMA box: row by row as bulk copies, or per thread by 8-byte copies, the issue alone
// costs 1,500-2,500 cycles a layer.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <atomic>
#include <type_traits>

#include "hm_async.cuh"
#include "hm_common.cuh"
#include "hm_internal.h"

namespace hm {

constexpr int kApplyThreads = 128;   // columns of a tile at most
constexpr int kApplyBlocks = 2;      // CTAs per SM in FP64 (8 warps, up to 255 registers)
constexpr int kApplyBlocks32 = 3;    // in FP32 (12 warps, up to 168; at four, 128, it spills: 38.5 against 33.1 us at 64^3)
constexpr int kApplyItems = 5;       // entries of a node plane per thread at most
constexpr int kRing = 6;             // node planes: a layer's two upper ones, four arriving

// what the input vector stands for: the vector itself (zero on the Dirichlet nodes), or the
// vector with the Dirichlet nodes zeroed on the fly
enum ApplyIn { IN_CLEAN = 0, IN_ESS = 1 };
// what is done with a node's product: y = A x (x itself on the Dirichlet nodes), a pass of
// the smoother (HmChebMode), or an assembled vector, y = A x - f int phi (0 on the Dirichlet
// nodes)
enum ApplyOut { OUT_Y = 0, OUT_R = 1, OUT_STEP1 = 2, OUT_START = 3, OUT_NEXT = 4, OUT_VEC = 5, OUT_POWER = 6 };

// the constant of HmCheb's kChebMax (cheb[1 + k]: c1_k, cheb[1 + kChebMax + k]: c2_k)
constexpr int kChebMax = 40;

// (a launch pays for the bytes of its parameters, ~0.1 us for 90: each kind of pass has its own)
template <typename src, typename vec>
struct ApplyArgs {
  const uint8_t* ess;
  const src* x;            // the input vector
  vec* y;                  // OUT_Y, OUT_VEC, OUT_POWER
  double* part;            // partial sums of x . y (OUT_Y) or b . z, one per CTA (NULL: none)
  double* sc;              // with part: the CG step's scalars (alpha or beta from the last block)
  unsigned* counter;
  double* fail;            // the solve's SC_FAIL (NULL: none)
  uint32_t* status;        // the library's status word (a bounded wait that gave up)
  int tma, pitch;          // D by TMA; its row pitch
};
// beside them for a pass of the smoother or of the power iteration
template <typename src, typename vec>
struct SmoothArgs : ApplyArgs<src, vec> {
  struct {                 // of HmCheb
    int k, first, last;
    const double *b, *idiag, *cheb;
    vec *x, *r, *dout;
    double* z;
  } c;
  const double* rr;        // beta: the partials of r.r
  unsigned nrr;
  int flex;
};
template <typename src, typename vec, int OUT>
using PassArgs = std::conditional_t<OUT == OUT_Y, ApplyArgs<src, vec>, SmoothArgs<src, vec>>;
// beside them for an assembled vector (OUT_VEC)
struct VecPart : ApplyArgs<double, double> {
  double sx, ry, rz;       // apply_tile's (computed there they take 2 us of 158 at 64^3; a small
                           // product is faster without the 24 bytes, 9.05 against 9.25 us at 12^3)
  uint32_t* caller;        // the caller's status word
  double f;                // the source, and int phi along each axis (phi_1d)
  double phi[3][3];
};

// ------------------------------------------------------------- 1D transforms
// nodes (x0, x1, x2) -> values at the points: 6 operations
template <typename T>
__device__ __forceinline__ void to_points(T x0, T x1, T x2, T& v0, T& v1, T& v2) {
  const T s = x0 + x2, d = x2 - x0;
  const T e = fma(T(0.4), x1, T(0.3) * s);
  v0 = fma(T(-kS), d, e);
  v1 = x1;
  v2 = fma(T(kS), d, e);
}
// values at the points -> derivatives there, times 2 sqrt(0.15): 5 operations
template <typename T>
__device__ __forceinline__ void derivs(T v0, T v1, T v2, T& g0, T& g1, T& g2) {
  const T d = v2 - v0;
  const T c = fma(T(-2), v1, v0 + v2);
  g0 = fma(T(-2), c, d);
  g1 = d;
  g2 = fma(T(2), c, d);
}
// the transposes: points -> nodes
template <typename T>
__device__ __forceinline__ void from_points(T f0, T f1, T f2, T& y0, T& y1, T& y2) {
  const T s = f0 + f2, m = f0 - f2;
  const T t = T(0.3) * s;
  y0 = fma(T(kS), m, t);
  y1 = fma(T(0.4), s, f1);
  y2 = fma(T(-kS), m, t);
}
// r += w (derivs transposed) f, with w4 = 4 w
template <typename T>
__device__ __forceinline__ void add_from_derivs(T f0, T f1, T f2, T w, T w4, T& r0, T& r1, T& r2) {
  const T m = f0 - f2;
  const T t = f1 + (f0 + f2);
  r0 = fma(-w, fma(T(2), m, t), r0);
  r1 = fma(w4, m, r1);
  r2 = fma(w, fma(T(-2), m, t), r2);
}

// int phi over its elements of a node's 1D basis function, on an axis of n elements: w[0] a
// middle node's, w[1] an end of the axis, w[2] between two elements
__device__ __forceinline__ double phi_1d(int i, int n, const double (&w)[3]) {
  return (i & 1) ? w[0] : (i == 0 || i == 2 * n) ? w[1] : w[2];
}

// A node plane at the element to its 9 points, less its middle node's value (x its first
// node, rows rs apart): each row less its own middle node first, whose value relative to the
// plane's goes in with the row's sum -- four operations more than the values themselves.
// Differences in the nodes' type, the rest in the arithmetic's.
template <typename T, typename src>
__device__ __forceinline__ void plane_to_points(const src* x, int rs, T (&v)[9]) {
  const src c = x[rs + 1];
  T r[9];
#pragma unroll
  for (int a2 = 0; a2 < 3; ++a2) {
    const src m = x[a2 * rs + 1];
    const T a = (T)(x[a2 * rs] - m), b = (T)(x[a2 * rs + 2] - m), w = a2 == 1 ? T(0) : (T)(m - c);
    const T d = b - a, t = fma(T(0.3), a + b, w);
    r[3 * a2] = fma(T(-kS), d, t);
    r[3 * a2 + 1] = w;
    r[3 * a2 + 2] = fma(T(kS), d, t);
  }
#pragma unroll
  for (int q1 = 0; q1 < 3; ++q1)
    to_points(r[q1], r[3 + q1], r[6 + q1], v[q1], v[3 + q1], v[6 + q1]);
}
// three planes' values along z, each less its own plane's reference r0, r1, r2, to the points
// less r1: k = 0.3 ((r0 - r1) + (r2 - r1)), g = r2 - r0
template <typename T>
__device__ __forceinline__ void to_points_z(T x0, T x1, T x2, T k, T g, T& v0, T& v1, T& v2) {
  const T d = (x2 - x0) + g;
  const T e = fma(T(0.4), x1, fma(T(0.3), x0 + x2, k));
  v0 = fma(T(-kS), d, e);
  v1 = x1;
  v2 = fma(T(kS), d, e);
}
template <typename T>
__device__ __forceinline__ void plane_from_points(T (&v)[9]) {
#pragma unroll
  for (int q1 = 0; q1 < 3; ++q1) from_points(v[q1], v[3 + q1], v[6 + q1], v[q1], v[3 + q1], v[6 + q1]);
#pragma unroll
  for (int a2 = 0; a2 < 3; ++a2)
    from_points(v[3 * a2], v[3 * a2 + 1], v[3 * a2 + 2], v[3 * a2], v[3 * a2 + 1], v[3 * a2 + 2]);
}
// One element at its 27 points: v0, v1, v2 the in-plane values of its three node planes (k, g:
// of to_points_z),
// D(q) the weights; on return the in-plane sums of the three planes
template <typename T, typename LDD>
__device__ __forceinline__ void element_points(T (&v0)[9], T (&v1)[9], T (&v2)[9], T k, T g, LDD D, T ry, T rz) {
  T V[27], R[27];          // [q1 + 3 q2 + 9 q3]
#pragma unroll
  for (int i = 0; i < 9; ++i) to_points_z(v0[i], v1[i], v2[i], k, g, V[i], V[9 + i], V[18 + i]);
#pragma unroll
  for (int i = 0; i < 9; ++i) {          // z lines
    T g0, g1, g2;
    derivs(V[i], V[9 + i], V[18 + i], g0, g1, g2);
    g0 *= D(i); g1 *= D(9 + i); g2 *= D(18 + i);
    R[i] = R[9 + i] = R[18 + i] = T(0);
    add_from_derivs(g0, g1, g2, rz, T(4) * rz, R[i], R[9 + i], R[18 + i]);
  }
#pragma unroll
  for (int q3 = 0; q3 < 3; ++q3) {       // x and y lines of slice q3
    T d[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) d[i] = D(9 * q3 + i);
#pragma unroll
    for (int q2 = 0; q2 < 3; ++q2) {
      const int i = 9 * q3 + 3 * q2;
      T g0, g1, g2;
      derivs(V[i], V[i + 1], V[i + 2], g0, g1, g2);
      add_from_derivs(g0 * d[3 * q2], g1 * d[3 * q2 + 1], g2 * d[3 * q2 + 2], T(1), T(4), R[i], R[i + 1], R[i + 2]);
    }
#pragma unroll
    for (int q1 = 0; q1 < 3; ++q1) {
      const int i = 9 * q3 + q1;
      T g0, g1, g2;
      derivs(V[i], V[i + 3], V[i + 6], g0, g1, g2);
      add_from_derivs(g0 * d[q1], g1 * d[3 + q1], g2 * d[6 + q1], ry, T(4) * ry, R[i], R[i + 3], R[i + 6]);
    }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) from_points(R[i], R[9 + i], R[18 + i], v0[i], v1[i], v2[i]);
}

// Loads where `on`, else 0, by a predicate and issued where they stand: with a branch around
// each, as conditional expressions and statements compile to here, a layer's loads and copies
// took 2,000 cycles to issue, with predicates 900 (16^3, y = A x alone: 9.8 -> 7.0 us in FP64,
// 11.9 -> 6.8 in FP32; 64^3 49.8 -> 38.8 and 57.2 -> 33.5).
__device__ __forceinline__ uint32_t load_mark(const uint8_t* p, bool on) {
  uint32_t m;
  asm volatile(
      "{\n .reg .pred p;\n .reg .u16 t;\n setp.ne.u32 p, %2, 0;\n mov.u16 t, 0;\n"
      " @p ld.global.nc.u8 t, [%1];\n cvt.u32.u16 %0, t;\n}"
      : "=r"(m)
      : "l"(p), "r"((uint32_t)on));
  return m;
}
// (not .nc: r and x are the kernel's own outputs too, node by node)
__device__ __forceinline__ double load_if(const double* p, bool on) {
  double v;
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.f64 %0, 0d0000000000000000;\n @p ld.global.f64 %0, [%1];\n}"
               : "=d"(v) : "l"(p), "r"((uint32_t)on) : "memory");
  return v;
}
__device__ __forceinline__ float load_if(const float* p, bool on) {
  float v;
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.f32 %0, 0f00000000;\n @p ld.global.f32 %0, [%1];\n}"
               : "=f"(v) : "l"(p), "r"((uint32_t)on) : "memory");
  return v;
}

// Dynamic shared memory: D of two layers [q][row][column] (one TMA box from the 16-byte
// boundary at or before the tile's first column), the ring of node planes, the exchange.
template <typename real> HM_HD constexpr int row_align() { return 16 / (int)sizeof(real); }
template <typename real>
HM_HD int box_columns(int T1) {
  constexpr int A = row_align<real>();
  return (T1 + 2 * A - 2) / A * A;
}
template <typename real, typename src>
struct ApplySmem {
  int dbuf, ring, exch, bytes;       // bytes of one D buffer, offsets in bytes
  HM_HD ApplySmem(const ApplyPlan& p) {
    const int s = (int)sizeof(real);
    dbuf = (27 * p.T2 * box_columns<real>(p.T1) * s + 127) / 128 * 128;
    ring = 2 * dbuf;
    exch = ring + kRing * (2 * p.T1 + 1) * (2 * p.T2 + 1) * (int)sizeof(src);
    bytes = exch + 20 * p.threads * s;
  }
};

// the work of one CTA, tile bt (D by the map at `map`)
template <typename real, typename src, typename vec, int IN, int OUT, typename Args>
__device__ __forceinline__ void apply_tile(const CUtensorMap* map, const Lattice& L, const real* __restrict__ Dq,
                                           const Args& a, const int bt) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ unsigned long long mbar[2];           // D of the even and the odd layers
  const ApplySmem<real, src> at(L.ap);
  constexpr int A = row_align<real>();
  const int T1 = L.ap.T1, T2 = L.ap.T2, nt = blockDim.x;
  src* const ring = reinterpret_cast<src*>(smem_raw + at.ring);
  real* const exch = reinterpret_cast<real*>(smem_raw + at.exch);
  const int RS = 2 * T1 + 1, P = RS * (2 * T2 + 1), TB = box_columns<real>(T1);
  const int tid = threadIdx.x;
  // the tile's first cells (a later tile's first column, row and layer are the halo)
  const int i1 = bt % L.ap.t1, i2 = (bt / L.ap.t1) % L.ap.t2, i3 = bt / (L.ap.t1 * L.ap.t2);
  const int c1 = i1 * (T1 - 1), c2 = i2 * (T2 - 1), c3 = i3 * (L.ap.T3 - 1);
  const int layers = min(L.ap.T3, L.nz + 1 - c3);
  const unsigned nsy = (unsigned)L.Nx, nsz = (unsigned)L.Nx * (unsigned)L.Ny;

  // ---- D of layer l (thread 0)
  auto request_D = [&](int l) {
    if (tid != 0 || !a.tma || l >= layers || c3 + l >= L.nz) return;
    fence_proxy_async();                   // the buffer's readers are done (block barrier)
    mbar_expect(&mbar[l & 1], 27u * (uint32_t)(T2 * TB) * (uint32_t)sizeof(real));
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(smem_raw + (l & 1) * at.dbuf)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c1 & ~(A - 1)), "r"(c2), "r"(c3 + l), "r"(0),
        "r"(smem_u32(&mbar[l & 1]))
        : "memory");
  };
  if (tid == 0) {
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
    fence_mbar_init();
  }
  request_D(0);
  request_D(1);
  // ---- node planes: plane j (relative to 2 c3) into ring slot j % kRing, entry i of a
  // plane by thread i % nt, the same ones every time
  unsigned off[kApplyItems];               // the entries' nodes in the mesh's plane (~0: none)
  {
    const int step_r = nt / RS, step_c = nt - step_r * RS;
    int r = tid / RS, c = tid - r * RS;
#pragma unroll
    for (int k = 0; k < kApplyItems; ++k) {
      const int gx = 2 * c1 + c, gy = 2 * c2 + r;
      off[k] = tid + k * nt < P && gx < L.Nx && gy < L.Ny ? (unsigned)gx + nsy * (unsigned)gy : ~0u;
      r += step_r;
      c += step_c;
      if (c >= RS) { c -= RS; ++r; }
    }
  }
  auto request = [&](int j) {
    if (2 * c3 + j < L.Nz && j <= 2 * layers) {
      src* const plane = ring + j % kRing * P + tid;
      const src* const x = a.x + (size_t)nsz * (2 * c3 + j);
#pragma unroll
      for (int k = 0; k < kApplyItems; ++k)
        if constexpr (OUT == OUT_VEC) {    // (a branch is the faster here, beside grad_tile: 158 us against 163 for three)
          if (off[k] != ~0u) copy_async(plane + k * nt, x + off[k], true);
        } else {
          copy_async(plane + k * nt, x + off[k], off[k] != ~0u);
        }
    }
  };
  // The Dirichlet markers of plane j are loaded a layer before finish() zeroes the marked
  // entries, after the plane's copies and by the same threads (loaded there, their latency
  // stood open twice a layer).
  struct Marks { uint32_t m[IN == IN_ESS ? kApplyItems : 1]; };
  auto load = [&](int j, Marks& e) {
    if constexpr (IN == IN_ESS) {
      const bool plane = a.ess != nullptr && 2 * c3 + j < L.Nz && j <= 2 * layers;
      const uint8_t* const ess = a.ess + (size_t)nsz * (2 * c3 + j);
#pragma unroll
      for (int k = 0; k < kApplyItems; ++k) e.m[k] = load_mark(ess + off[k], plane && off[k] != ~0u);
    }
  };
  auto finish = [&](int j, const Marks& e) {
    if constexpr (IN == IN_ESS) {
      src* const plane = ring + j % kRing * P + tid;
#pragma unroll
      for (int k = 0; k < kApplyItems; ++k)
        if (e.m[k] != 0u) plane[k * nt] = src(0);
    }
  };
  // D is requested a layer ahead, node planes two layers, a group of copies each
  for (int j = 0; j < 3; ++j) request(j);
  copy_commit();
  request(3);
  request(4);
  copy_commit();
  const int ty = tid / T1, tx = tid - ty * T1;
  const int cx = c1 + tx, cy = c2 + ty;
  const bool column = ty < T2;
  const bool element = column && cx < L.nx && cy < L.ny;
  const bool own = column && cx <= L.nx && cy <= L.ny && (tx > 0 || i1 == 0) && (ty > 0 || i2 == 0);
  double inv_theta = 0.0;
  if constexpr (OUT == OUT_STEP1 || OUT == OUT_START) inv_theta = 1.0 / __ldg(a.c.cheb);
  double w1 = 0.0, w2 = 0.0;               // step k: dout = w1 in + w2 r idiag
  if constexpr (OUT == OUT_NEXT) {
    w1 = __ldg(a.c.cheb + 1 + a.c.k);
    w2 = __ldg(a.c.cheb + 1 + kChebMax + a.c.k);
  }
  {
    Marks e[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) load(j, e[j]);
    copy_wait<1>();
#pragma unroll
    for (int j = 0; j < 3; ++j) finish(j, e[j]);
  }
  __syncthreads();

  // the product's scale (the derivatives carry 2 sqrt(0.15) each: 1 / (4 * 0.15) in the product),
  // the weights of the y and z derivatives in it
  real sx, ry, rz;
  if constexpr (OUT == OUT_VEC) {
    sx = a.sx; ry = a.ry; rz = a.rz;
  } else {
    sx = (real)(1.0 / (0.6 * L.hx * L.hx));
    ry = (real)((L.hx * L.hx) / (L.hy * L.hy));
    rz = (real)((L.hx * L.hx) / (L.hz * L.hz));
  }
  const int base = 2 * ty * RS + 2 * tx;  // the element's first node in a plane
  // in-plane values of the lower node plane less its middle node's, that value, sums of the
  // lower layer on it, the input at the own nodes there.  (The operator annihilates
  // constants: values at the points that carried the field's own would give every
  // derivative the field's rounding over h.)
  real low[9], carry[9];
  src clow = src(0), xlow[4];
#pragma unroll
  for (int i = 0; i < 9; ++i) low[i] = carry[i] = real(0);
  if (element) {
    clow = ring[base + RS + 1];
    plane_to_points(ring + base, RS, low);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) xlow[k] = own ? ring[base + (k >> 1) * RS + (k & 1)] : src(0);
  __syncthreads();                        // plane 0's slot is plane 6's, requested next
  double dot = 0.0;
#pragma unroll 1
  for (int l = 0; l < layers; ++l) {
    const int cz = c3 + l;
    const src* const p1 = ring + (2 * l + 1) % kRing * P + base;
    const src* const p2 = ring + (2 * l + 2) % kRing * P + base;
    // The own nodes h = (x, y, z parity bits): which of them exist, their markers
    // (requested here, used after the barrier)
    const bool out = own && (l > 0 || i3 == 0);
    const unsigned n0 = (unsigned)(2 * cx) + nsy * (unsigned)(2 * cy) + nsz * (unsigned)(2 * cz);
    unsigned have = 0;
    if (out) have = 0x55u | (cx < L.nx ? 0xaau : 0u);
    if (cy >= L.ny) have &= 0x33u;
    if (cz >= L.nz) have &= 0x0fu;
    uint32_t mark[8];
    // (left to the compiler where the pass loads nothing else by predicate: CG's product at
    // 64^3 40.2 us against 41.0, dR/du 68 against 70)
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      const unsigned node = n0 + (h & 1) + ((h & 2) ? nsy : 0u) + ((h & 4) ? nsz : 0u);
      const bool on = a.ess != nullptr && ((have >> h) & 1u);
      if constexpr (IN == IN_CLEAN && (OUT == OUT_Y || OUT == OUT_VEC)) mark[h] = on ? __ldg(a.ess + node) : 0u;
      else mark[h] = load_mark(a.ess + node, on);
    }
    request(2 * l + 5);
    request(2 * l + 6);
    copy_commit();
    if (l > 0) request_D(l + 1);
    Marks next[2];
    load(2 * l + 3, next[0]);
    load(2 * l + 4, next[1]);
    real y[18];                            // the element's sums on its two lower planes
    const bool layer = cz < L.nz;          // not the virtual one
    const bool ok = !a.tma || !layer || mbar_wait(&mbar[l & 1], (uint32_t)(l >> 1) & 1u);
    if (element && layer) {
      const int ds = T2 * TB;
      real* const Dl = reinterpret_cast<real*>(smem_raw + (l & 1) * at.dbuf) + ty * TB + tx + (c1 & (A - 1));
      if (!a.tma) {                        // storage without a 16-byte pitch: this thread's own
        const real* const Dg = Dq + (size_t)cx + (size_t)a.pitch * ((size_t)cy + (size_t)L.ny * (size_t)cz);
#pragma unroll 1
        for (int q = 0; q < 27; q += 9) {
          real v[9];
#pragma unroll
          for (int i = 0; i < 9; ++i) v[i] = __ldg(Dg + (size_t)(q + i) * a.pitch * L.ny * L.nz);
#pragma unroll
          for (int i = 0; i < 9; ++i) Dl[(q + i) * ds] = v[i];
        }
      }
      real v1[9], v2[9];
      plane_to_points(p1, RS, v1);
      plane_to_points(p2, RS, v2);
      real up[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) up[i] = v2[i];
      const src mid = p1[RS + 1], cup = p2[RS + 1];
      const real k = real(0.3) * (real)((clow - mid) + (cup - mid)), g = (real)(cup - clow);
      clow = cup;
      element_points(low, v1, v2, k, g, [&](int q) { return Dl[q * ds]; }, ry, rz);
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        low[i] += carry[i];
        carry[i] = v2[i];
      }
      plane_from_points(low);
      plane_from_points(v1);
#pragma unroll
      for (int i = 0; i < 9; ++i) { y[i] = low[i]; y[9 + i] = v1[i]; low[i] = up[i]; }
    } else {
      plane_from_points(carry);
#pragma unroll
      for (int i = 0; i < 9; ++i) { y[i] = carry[i]; y[9 + i] = carry[i] = real(0); }
    }
    // (keeps the markers' first use here, after the arithmetic)
#pragma unroll
    for (int h = 0; h < 8; ++h) asm volatile("" : "+r"(mark[h]));
    // the results other columns' nodes need: a1 = 2 (a2 = 0, 1, 2), a2 = 2 (a1 = 0, 1)
    real* const ex = exch + (l & 1) * 10 * nt;
#pragma unroll
    for (int a3 = 0; a3 < 2; ++a3) {
      real* const e = ex + a3 * 5 * nt + tid;
      e[0] = y[9 * a3 + 2];
      e[nt] = y[9 * a3 + 5];
      e[2 * nt] = y[9 * a3 + 8];
      e[3 * nt] = y[9 * a3 + 6];
      e[4 * nt] = y[9 * a3 + 7];
    }
    // the input at the own nodes (the zeroed ones' too), the smoother's operands
    src xc[8];
    double bn[OUT == OUT_Y || OUT == OUT_VEC || OUT == OUT_POWER ? 1 : 8], gn[OUT == OUT_Y || OUT == OUT_R || OUT == OUT_VEC ? 1 : 8], xn[OUT == OUT_NEXT ? 8 : 1];
    unsigned fixed = 0;
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      const bool on = (have >> h) & 1u;
      const unsigned node = n0 + (h & 1) + ((h & 2) ? nsy : 0u) + ((h & 4) ? nsz : 0u);
      if constexpr (OUT == OUT_NEXT) {
        if (a.c.first) bn[h] = load_if(a.c.b + node, on);
        else bn[h] = (double)load_if(a.c.r + node, on);
        xn[h] = (double)load_if(a.c.x + node, on && !a.c.first);
      } else if constexpr (OUT != OUT_Y && OUT != OUT_VEC && OUT != OUT_POWER) {
        bn[h] = load_if(a.c.b + node, on);
      }
      if constexpr (OUT != OUT_Y && OUT != OUT_R && OUT != OUT_VEC) gn[h] = load_if(a.c.idiag + node, on);
      const int o = ((h >> 1) & 1) * RS + (h & 1);
      if (h < 4) {
        xc[h] = xlow[h];
        xlow[h] = own ? p2[o] : src(0);
      } else {
        xc[h] = own ? p1[o] : src(0);
      }
      fixed |= (unsigned)(mark[h] != 0u) << h;
      if constexpr (IN == IN_ESS)
        if (on && mark[h] != 0u) xc[h] = __ldg(a.x + node);
    }
    copy_wait<1>();                        // the next layer's planes
    finish(2 * l + 3, next[0]);
    finish(2 * l + 4, next[1]);
    if (__syncthreads_or(!ok || L.give_up)) {   // a copy never landed: flagged, nothing more written
      if (tid == 0) {
        if (a.status != nullptr) atomicOr(a.status, HM_STATUS_TIMEOUT);
        if constexpr (OUT == OUT_VEC) atomicOr(a.caller, HM_STATUS_TIMEOUT);
        else if (a.fail != nullptr) *a.fail = 1.0;
        // both buffers' copies, before the CTA leaves
        (void)mbar_wait(&mbar[l & 1], (uint32_t)(l >> 1) & 1u);
        if (l + 1 < layers && cz + 1 < L.nz) (void)mbar_wait(&mbar[(l + 1) & 1], (uint32_t)((l + 1) >> 1) & 1u);
      }
      break;
    }
    if (have) {
      const bool left = tx > 0, front = ty > 0;
#pragma unroll
      for (int a3 = 0; a3 < 2; ++a3) {
        const real* const e = ex + a3 * 5 * nt + tid;
        real n[4];                        // nodes (0,0), (1,0), (0,1), (1,1)
        n[0] = y[9 * a3]; n[1] = y[9 * a3 + 1]; n[2] = y[9 * a3 + 3]; n[3] = y[9 * a3 + 4];
        if (left) { n[0] += e[-1]; n[2] += e[nt - 1]; }
        if (front) { n[0] += e[3 * nt - T1]; n[1] += e[4 * nt - T1]; }
        if (left && front) n[0] += e[2 * nt - T1 - 1];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int h = 4 * a3 + k;
          if (!((have >> h) & 1u)) continue;
          const unsigned node = n0 + (k & 1) + ((k & 2) ? nsy : 0u) + (a3 ? nsz : 0u);
          const bool fx = (fixed >> h) & 1u;
          const double acc = (double)(sx * n[k]);
          if constexpr (OUT == OUT_Y) {
            const double xv = (double)xc[h];
            const double yv = fx ? xv : acc;
            a.y[node] = (vec)yv;
            dot = fma(xv, yv, dot);
          } else if constexpr (OUT == OUT_VEC) {
            double v = acc;
            if (a.f != 0.0)
              v -= a.f * (phi_1d(2 * cx + (k & 1), L.nx, a.phi[0]) * phi_1d(2 * cy + (k >> 1), L.ny, a.phi[1]) *
                          phi_1d(2 * cz + a3, L.nz, a.phi[2]));
            a.y[node] = (vec)(fx ? 0.0 : v);
          } else if constexpr (OUT == OUT_POWER) {
            a.y[node] = (vec)(fx ? 0.0 : acc * gn[h]);
          } else {
            const double in = (double)xc[h];
            const double ri = bn[h] - (fx ? in : acc);
            if constexpr (OUT == OUT_R) {
              a.c.r[node] = (vec)ri;
            } else if constexpr (OUT == OUT_STEP1) {
              // the update rounded on its own before the add, as the step-by-step smoother
              const double z = in + __dmul_rn(inv_theta * ri, gn[h]);
              a.c.z[node] = z;
              dot = fma(bn[h], z, dot);
            } else if constexpr (OUT == OUT_START) {
              a.c.r[node] = (vec)ri;
              a.c.dout[node] = (vec)(inv_theta * ri * gn[h]);
            } else {
              const double xi = a.c.first ? in : xn[h] + in;
              const double dn = fma(w1, in, w2 * ri * gn[h]);
              if (a.c.last == 2) {
                const double z = xi + dn;
                a.c.z[node] = z;
                if (a.part != nullptr) dot = fma(__ldg(a.c.b + node), z, dot);
              } else {
                a.c.x[node] = (vec)xi;
                a.c.r[node] = (vec)ri;
                if (a.c.last == 0) a.c.dout[node] = (vec)dn;
              }
            }
          }
        }
      }
    }
  }
  copy_wait<0>();
  if constexpr (OUT != OUT_R && OUT != OUT_START && OUT != OUT_VEC && OUT != OUT_POWER) {
    if (a.part != nullptr) {
      __shared__ double sh[32];
      const double t = block_sum(dot, sh);
      if (tid == 0) a.part[blockIdx.x] = t;
      // a CG step: the last block takes alpha, or beta, from the partials
      if (a.sc != nullptr && last_block(a.counter)) {
        if constexpr (OUT == OUT_Y) finish_alpha(a.part, gridDim.x, a.sc, a.counter, sh);
        else finish_beta(a.part, gridDim.x, a.rr, a.nrr, a.flex, a.sc, a.counter, sh);
      }
    }
  }
}

template <typename real, typename src, typename vec, int IN, int OUT>
__global__ void __launch_bounds__(kApplyThreads, sizeof(real) == 8 ? kApplyBlocks : kApplyBlocks32)
    k_apply_tile(const __grid_constant__ CUtensorMap map, const Lattice L, const real* __restrict__ Dq,
                 const PassArgs<src, vec, OUT> a) {
  apply_tile<real, src, vec, IN, OUT>(&map, L, Dq, a, (int)blockIdx.x);
}

// ------------------------------------------------------------ assembled vectors
// dR/dp (ADJOINT, with the source) is A(D) u, dR/du (STATE) is A(D) p, both without
// elimination: apply_tile.  dR/dm (PARAMETER) integrates W = D grad u . grad p against the
// basis: grad_tile.  With mhat, D = w|J| e^m mhat and these are the second-order products
// along mhat.  Bound: FP64 arithmetic (27 exponentials, then ~680 operations an element and
// vector), D through memory once between the two launches.  Measured at 64^3: three vectors
// 152 us (D 28; 163 with L2 flushed before), the gradient alone 73; at 32^3 44 and 19, at
// 16^3 14 and 11, against 486 (499) and 381, 68 and 53, 19 and 12 us for an element pass
// whose stages all go through shared memory and a node gather per vector.

// D at the points of every element (a thread each), and the check that every pointwise value
// the vectors are made of (E = D grad u, F = D grad p, W) is finite: by bounds on the nodes'
// values, and only where those do not settle it by the values themselves.
__global__ void __launch_bounds__(128)
    k_points_D(const Lattice L, int pitch, const double* __restrict__ u, const double* __restrict__ m,
               const double* __restrict__ p, const double* __restrict__ mhat, double* __restrict__ D,
               uint32_t* __restrict__ status, const uint32_t* __restrict__ skip) {
  if (skip != nullptr && *skip != 0u) return;
  const unsigned e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (unsigned)L.ne) return;
  const unsigned row = e / (unsigned)L.nx, ex = e - row * (unsigned)L.nx;
  const unsigned ez = row / (unsigned)L.ny, ey = row - ez * (unsigned)L.ny;
  const unsigned nsy = (unsigned)L.Nx, nsz = nsy * (unsigned)L.Ny;
  const unsigned n0 = 2u * ex + nsy * 2u * ey + nsz * 2u * ez;
  auto load = [&](const double* x, double (&v)[27]) {
#pragma unroll
    for (int i = 0; i < 27; ++i) v[i] = __ldg(x + n0 + (unsigned)(i % 3) + nsy * (unsigned)((i / 3) % 3) + nsz * (unsigned)(i / 9));
  };
  auto points = [&](double (&v)[27]) {       // node values to point values, in place
#pragma unroll
    for (int i = 0; i < 9; ++i) to_points(v[3 * i], v[3 * i + 1], v[3 * i + 2], v[3 * i], v[3 * i + 1], v[3 * i + 2]);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const int o = (i / 3) * 9 + i % 3;
      to_points(v[o], v[o + 3], v[o + 6], v[o], v[o + 3], v[o + 6]);
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) to_points(v[i], v[9 + i], v[18 + i], v[i], v[9 + i], v[18 + i]);
  };
  double d[27];
  load(m, d);
  points(d);
  const double vol = L.hx * L.hy * L.hz;
#pragma unroll
  for (int q = 0; q < 27; ++q) d[q] = wq(q % 3) * wq((q / 3) % 3) * wq(q / 9) * vol * exp(d[q]);
  if (mhat != nullptr) {
    double h[27];
    load(mhat, h);
    points(h);
#pragma unroll
    for (int q = 0; q < 27; ++q) d[q] *= h[q];
  }
  double* const out = D + ex + (size_t)pitch * row;
  const size_t dq = (size_t)pitch * L.ny * L.nz;
  double dmax = 0.0;
  bool bad = false;
#pragma unroll
  for (int q = 0; q < 27; ++q) {
    out[q * dq] = d[q];
    bad |= !(fabs(d[q]) < 1e290);
    dmax = fmax(dmax, fabs(d[q]));
  }
  double umax = 0.0, pmax = 0.0, v[27];
  load(u, v);
#pragma unroll
  for (int i = 0; i < 27; ++i) { bad |= !(fabs(v[i]) < 1e290); umax = fmax(umax, fabs(v[i])); }
  load(p, v);
#pragma unroll
  for (int i = 0; i < 27; ++i) { bad |= !(fabs(v[i]) < 1e290); pmax = fmax(pmax, fabs(v[i])); }
  // |grad| <= c max|.| per component: the derivative's absolute row sum is at most 8 / h, the
  // values' at most 1.6 on either other axis
  const double c = 24.0 * fmax(1.0 / L.hx, fmax(1.0 / L.hy, 1.0 / L.hz));
  const double gu = c * umax, gp = c * pmax;
  if (!bad && dmax * gu < 1e290 && dmax * gp < 1e290 && gu * gp < 1e290 && dmax * (3.0 * gu * gp) < 1e290) return;
  // the values themselves
#pragma unroll 1
  for (int q = 0; q < 27; ++q) {
    const int q1 = q % 3, q2 = (q / 3) % 3, q3 = q / 9;
    double gr[2][3] = {{0, 0, 0}, {0, 0, 0}};
#pragma unroll 1
    for (int i = 0; i < 27; ++i) {
      const unsigned n = n0 + (unsigned)(i % 3) + nsy * (unsigned)((i / 3) % 3) + nsz * (unsigned)(i / 9);
      const double b1 = bq(q1, i % 3), b2 = bq(q2, (i / 3) % 3), b3 = bq(q3, i / 9);
      const double x = dbq(q1, i % 3) * b2 * b3, y = b1 * dbq(q2, (i / 3) % 3) * b3, z = b1 * b2 * dbq(q3, i / 9);
      for (int k = 0; k < 2; ++k) {
        const double val = k == 0 ? u[n] : p[n];
        gr[k][0] = fma(x, val, gr[k][0]); gr[k][1] = fma(y, val, gr[k][1]); gr[k][2] = fma(z, val, gr[k][2]);
      }
    }
    const double dv = out[q * dq];
    double dot = 0.0;
    bool fine = true;
    for (int k = 0; k < 3; ++k) {
      const double h = k == 0 ? L.hx : k == 1 ? L.hy : L.hz;
      const double a = gr[0][k] / h, b = gr[1][k] / h;
      fine = fine && isfinite(dv * a) && isfinite(dv * b);
      dot += a * b;
    }
    if (!(fine && isfinite(dv * dot))) {
      atomicOr(status, HM_STATUS_NONFINITE);
      return;
    }
  }
}

// dR/dm: a tile of columns marching up z as in apply_tile, for two vectors.  The in-plane
// values of a layer's lower node plane are formed again from the ring (both vectors' would
// be 36 registers more); D is needed only at the end of a layer's arithmetic and has one
// buffer.
constexpr int kGradRing = 5;         // a layer's three planes, two arriving
struct GradSmem {
  int ring, exch, bytes;
  HM_HD GradSmem(const ApplyPlan& p) {
    ring = (27 * p.T2 * box_columns<double>(p.T1) * 8 + 127) / 128 * 128;
    exch = ring + 2 * kGradRing * (2 * p.T1 + 1) * (2 * p.T2 + 1) * 8;
    bytes = exch + 20 * p.threads * 8;
  }
};
__device__ __forceinline__ void grad_tile(const CUtensorMap* map, const Lattice& L, const double* __restrict__ Dq,
                                          int tma, int pitch, const double* __restrict__ u,
                                          const double* __restrict__ p, double* __restrict__ yout,
                                          const VecPart& a, const int bt) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ unsigned long long mbar;
  const GradSmem at(L.ap);
  const int T1 = L.ap.T1, T2 = L.ap.T2, nt = blockDim.x;
  double* const ring = reinterpret_cast<double*>(smem_raw + at.ring);
  double* const exch = reinterpret_cast<double*>(smem_raw + at.exch);
  const int RS = 2 * T1 + 1, P = RS * (2 * T2 + 1), TB = box_columns<double>(T1);
  const int tid = threadIdx.x;
  const int i1 = bt % L.ap.t1, i2 = (bt / L.ap.t1) % L.ap.t2, i3 = bt / (L.ap.t1 * L.ap.t2);
  const int c1 = i1 * (T1 - 1), c2 = i2 * (T2 - 1), c3 = i3 * (L.ap.T3 - 1);
  const int layers = min(L.ap.T3, L.nz + 1 - c3);
  const unsigned nsy = (unsigned)L.Nx, nsz = (unsigned)L.Nx * (unsigned)L.Ny;
  auto request_D = [&](int l) {
    if (tid != 0 || !tma || l >= layers || c3 + l >= L.nz) return;
    fence_proxy_async();                   // the buffer's readers are done (block barrier)
    mbar_expect(&mbar, 27u * (uint32_t)(T2 * TB) * 8u);
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(smem_raw)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c1 & ~1), "r"(c2), "r"(c3 + l), "r"(0),
        "r"(smem_u32(&mbar))
        : "memory");
  };
  if (tid == 0) {
    mbar_init(&mbar, 1);
    fence_mbar_init();
  }
  request_D(0);
  unsigned off[kApplyItems];               // as in apply_tile
  {
    const int step_r = nt / RS, step_c = nt - step_r * RS;
    int r = tid / RS, c = tid - r * RS;
#pragma unroll
    for (int k = 0; k < kApplyItems; ++k) {
      const int gx = 2 * c1 + c, gy = 2 * c2 + r;
      off[k] = tid + k * nt < P && gx < L.Nx && gy < L.Ny ? (unsigned)gx + nsy * (unsigned)gy : ~0u;
      r += step_r;
      c += step_c;
      if (c >= RS) { c -= RS; ++r; }
    }
  }
  auto request = [&](int j) {
    if (2 * c3 + j < L.Nz && j <= 2 * layers) {
      double* const pu = ring + j % kGradRing * P + tid;
      const size_t z0 = (size_t)nsz * (2 * c3 + j);
#pragma unroll
      for (int k = 0; k < kApplyItems; ++k) {
        copy_async(pu + k * nt, u + z0 + off[k], off[k] != ~0u);
        copy_async(pu + kGradRing * P + k * nt, p + z0 + off[k], off[k] != ~0u);
      }
    }
  };
  for (int j = 0; j < 3; ++j) request(j);
  copy_commit();
  const int ty = tid / T1, tx = tid - ty * T1;
  const int cx = c1 + tx, cy = c2 + ty;
  const bool column = ty < T2;
  const bool element = column && cx < L.nx && cy < L.ny;
  const bool own = column && cx <= L.nx && cy <= L.ny && (tx > 0 || i1 == 0) && (ty > 0 || i2 == 0);
  const double sx = a.sx, ry = a.ry, rz = a.rz;
  const int base = 2 * ty * RS + 2 * tx, ds = T2 * TB;
  double carry[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) carry[i] = 0.0;
  copy_wait<0>();
  __syncthreads();
#pragma unroll 1
  for (int l = 0; l < layers; ++l) {
    const int cz = c3 + l;
    const double* const p0 = ring + (2 * l) % kGradRing * P + base;
    const double* const p1 = ring + (2 * l + 1) % kGradRing * P + base;
    const double* const p2 = ring + (2 * l + 2) % kGradRing * P + base;
    request(2 * l + 3);
    request(2 * l + 4);
    copy_commit();
    if (l > 0) request_D(l);
    const bool layer = cz < L.nz;
    bool ok = true;
    double y[18];
    if (element && layer) {
      double* const Dl = reinterpret_cast<double*>(smem_raw) + ty * TB + tx + (c1 & 1);
      if (!tma) {
        const double* const Dg = Dq + (size_t)cx + (size_t)pitch * ((size_t)cy + (size_t)L.ny * (size_t)cz);
#pragma unroll 1
        for (int q = 0; q < 27; q += 9) {
          double v[9];
#pragma unroll
          for (int i = 0; i < 9; ++i) v[i] = __ldg(Dg + (size_t)(q + i) * pitch * L.ny * L.nz);
#pragma unroll
          for (int i = 0; i < 9; ++i) Dl[(q + i) * ds] = v[i];
        }
      }
      double U[27], Q[27], W[27];
      auto values = [&](int o, double (&V)[27]) {
        double v0[9], v1[9], v2[9];
        plane_to_points(p0 + o, RS, v0);
        plane_to_points(p1 + o, RS, v1);
        plane_to_points(p2 + o, RS, v2);
        const double r0 = p0[o + RS + 1], r1 = p1[o + RS + 1], r2 = p2[o + RS + 1];
        const double k = 0.3 * ((r0 - r1) + (r2 - r1)), g = r2 - r0;
#pragma unroll
        for (int i = 0; i < 9; ++i) to_points_z(v0[i], v1[i], v2[i], k, g, V[i], V[9 + i], V[18 + i]);
      };
      values(0, U);
      values(kGradRing * P, Q);
      auto line = [&](int a, int b, int c, double w, bool first) {
        double g0, g1, g2, h0, h1, h2;
        derivs(U[a], U[b], U[c], g0, g1, g2);
        derivs(Q[a], Q[b], Q[c], h0, h1, h2);
        h0 *= w; h1 *= w; h2 *= w;
        W[a] = first ? g0 * h0 : fma(g0, h0, W[a]);
        W[b] = first ? g1 * h1 : fma(g1, h1, W[b]);
        W[c] = first ? g2 * h2 : fma(g2, h2, W[c]);
      };
#pragma unroll
      for (int i = 0; i < 9; ++i) line(i, 9 + i, 18 + i, rz, true);
#pragma unroll
      for (int i = 0; i < 9; ++i) line((i / 3) * 9 + i % 3, (i / 3) * 9 + i % 3 + 3, (i / 3) * 9 + i % 3 + 6, ry, false);
#pragma unroll
      for (int i = 0; i < 9; ++i) line(3 * i, 3 * i + 1, 3 * i + 2, 1.0, false);
      ok = !tma || mbar_wait(&mbar, (uint32_t)l & 1u);
#pragma unroll
      for (int q = 0; q < 27; ++q) W[q] *= Dl[q * ds];
      double m0[9], m1[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        double m2;
        from_points(W[i], W[9 + i], W[18 + i], m0[i], m1[i], m2);
        m0[i] += carry[i];
        carry[i] = m2;
      }
      plane_from_points(m0);
      plane_from_points(m1);
#pragma unroll
      for (int i = 0; i < 9; ++i) { y[i] = m0[i]; y[9 + i] = m1[i]; }
    } else {
      // every thread sees the layer's copy land before its buffer is requested again
      ok = !tma || !layer || mbar_wait(&mbar, (uint32_t)l & 1u);
      plane_from_points(carry);
#pragma unroll
      for (int i = 0; i < 9; ++i) { y[i] = carry[i]; y[9 + i] = carry[i] = 0.0; }
    }
    double* const ex = exch + (l & 1) * 10 * nt;
#pragma unroll
    for (int a3 = 0; a3 < 2; ++a3) {
      double* const e = ex + a3 * 5 * nt + tid;
      e[0] = y[9 * a3 + 2];
      e[nt] = y[9 * a3 + 5];
      e[2 * nt] = y[9 * a3 + 8];
      e[3 * nt] = y[9 * a3 + 6];
      e[4 * nt] = y[9 * a3 + 7];
    }
    copy_wait<0>();                        // the next layer's planes
    if (__syncthreads_or(!ok || L.give_up)) {
      if (tid == 0) {
        if (a.status != nullptr) atomicOr(a.status, HM_STATUS_TIMEOUT);
        atomicOr(a.caller, HM_STATUS_TIMEOUT);
        (void)mbar_wait(&mbar, (uint32_t)l & 1u);        // the copy, before the CTA leaves
      }
      break;
    }
    if (own && (l > 0 || i3 == 0)) {
      const bool left = tx > 0, front = ty > 0;
      const unsigned n0 = (unsigned)(2 * cx) + nsy * (unsigned)(2 * cy) + nsz * (unsigned)(2 * cz);
#pragma unroll
      for (int a3 = 0; a3 < 2; ++a3) {
        if (a3 == 1 && !layer) break;
        const double* const e = ex + a3 * 5 * nt + tid;
        double n[4];
        n[0] = y[9 * a3]; n[1] = y[9 * a3 + 1]; n[2] = y[9 * a3 + 3]; n[3] = y[9 * a3 + 4];
        if (left) { n[0] += e[-1]; n[2] += e[nt - 1]; }
        if (front) { n[0] += e[3 * nt - T1]; n[1] += e[4 * nt - T1]; }
        if (left && front) n[0] += e[2 * nt - T1 - 1];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (!((k & 1) && cx >= L.nx) && !((k & 2) && cy >= L.ny))
            yout[n0 + (k & 1) + ((k & 2) ? nsy : 0u) + (a3 ? nsz : 0u)] = sx * n[k];
      }
    }
  }
  copy_wait<0>();
}

// The requested vectors in one launch: `count` CTAs in a row take one tile's vectors, so
// that its D comes from memory once.
struct VecArgs {
  VecPart a[2];                        // ADJOINT, STATE
  const double* u;
  const double* p;
  double* grad;                        // PARAMETER
  int which[3], count;                 // 0, 1: a[which]; 2: grad
  const uint32_t* skip;                // nonzero there: the whole launch stands down
};
__global__ void __launch_bounds__(kApplyThreads, 2)
    k_vectors(const __grid_constant__ CUtensorMap map, const Lattice L, const double* __restrict__ D,
              const __grid_constant__ VecArgs v) {
  if (v.skip != nullptr && *v.skip != 0u) return;
  const int bt = (int)blockIdx.x / v.count, w = v.which[(int)blockIdx.x - bt * v.count];
  if (w == 2) grad_tile(&map, L, D, v.a[0].tma, v.a[0].pitch, v.u, v.p, v.grad, v.a[0], bt);
  else apply_tile<double, double, double, IN_CLEAN, OUT_VEC>(&map, L, D, v.a[w], bt);
}

// b . z and the CG step's beta on their own, after a cycle that ends in another kernel: the
// sum in k_apply_tile's order (a thread's own nodes layer by layer), so that a solve does
// not depend on which of the two took it
__global__ void __launch_bounds__(kApplyThreads)
    k_tile_beta(const Lattice L, const double* __restrict__ b, const double* __restrict__ z, HmBeta be) {
  __shared__ double sh[32];
  const int T1 = L.ap.T1, T2 = L.ap.T2, bt = blockIdx.x;
  const int i1 = bt % L.ap.t1, i2 = (bt / L.ap.t1) % L.ap.t2, i3 = bt / (L.ap.t1 * L.ap.t2);
  const int ty = threadIdx.x / T1, tx = threadIdx.x - ty * T1;
  const int cx = i1 * (T1 - 1) + tx, cy = i2 * (T2 - 1) + ty, c3 = i3 * (L.ap.T3 - 1);
  const bool own = ty < T2 && cx <= L.nx && cy <= L.ny && (tx > 0 || i1 == 0) && (ty > 0 || i2 == 0);
  const int layers = min(L.ap.T3, L.nz + 1 - c3);
  double dot = 0.0;
  if (own)
    for (int l = i3 == 0 ? 0 : 1; l < layers; ++l)
      for (int h = 0; h < 8; ++h) {
        const int x = 2 * cx + (h & 1), y = 2 * cy + ((h >> 1) & 1), w = 2 * (c3 + l) + (h >> 2);
        if (x >= L.Nx || y >= L.Ny || w >= L.Nz) continue;
        const int64_t n = x + (int64_t)L.Nx * (y + (int64_t)L.Ny * w);
        dot = fma(b[n], z[n], dot);
      }
  const double t = block_sum(dot, sh);
  if (threadIdx.x == 0) be.rz[blockIdx.x] = t;
  if (last_block(be.counter)) finish_beta(be.rz, gridDim.x, be.rr, be.n, be.flex, be.sc, be.counter, sh);
}

}  // namespace hm

using namespace hm;

// ------------------------------------------------------------------ host side
// The tiling: t_d tiles of T_d cells along axis d (the first owns T_d cells, the others
// T_d - 1 and the halo cell below), at most kApplyThreads columns.  Estimated time: a
// layer of a warp takes its arithmetic's share of the SM (4 warps of the CTAs on an SM
// progress together), or at least its own latency, with two CTAs resident per SM.
constexpr double kWarpLayer = 0.31, kLayer = 2.2, kStart = 4.5;   // us, measured
void hm_plan_apply(Lattice* L) {
  const int n[3] = {L->nx, L->ny, L->nz};
  double best = 0.0;
  ApplyPlan p{};
  int seen1 = 0;
  for (int t1 = 1; t1 <= n[0]; ++t1) {
    const int T1 = (n[0] + t1 - 1) / t1 + 1;
    if (T1 == seen1) continue;
    seen1 = T1;
    int seen2 = 0;
    for (int t2 = 1; t2 <= n[1]; ++t2) {
      const int T2 = (n[1] + t2 - 1) / t2 + 1;
      if (T2 == seen2) continue;
      seen2 = T2;
      const int warps = (T1 * T2 + 31) / 32;
      if (T1 * T2 > kApplyThreads || (2 * T1 + 1) * (2 * T2 + 1) > kApplyItems * 32 * warps) continue;
      int seen3 = 0;
      for (int t3 = 1; t3 <= n[2]; ++t3) {
        const int T3 = (n[2] + t3 - 1) / t3 + 1;
        if (T3 == seen3) continue;
        seen3 = T3;
        const int a1 = (n[0] + T1 - 2) / (T1 - 1), a2 = (n[1] + T2 - 2) / (T2 - 1),
                  a3 = (n[2] + T3 - 2) / (T3 - 1);
        const int64_t ctas = (int64_t)a1 * a2 * a3;
        const int64_t per_sm = (ctas + 147) / 148;
        const int resident = per_sm < kApplyBlocks ? (int)per_sm : kApplyBlocks;
        const double waves = (double)((per_sm + resident - 1) / resident);
        const double layer = resident * warps * kWarpLayer;
        const double cost = waves * (T3 * (layer > kLayer ? layer : kLayer) + kStart);
        if (p.threads == 0 || cost < best) {
          best = cost;
          p.T1 = T1; p.T2 = T2; p.T3 = T3;
          p.t1 = a1; p.t2 = a2; p.t3 = a3;
          p.threads = 32 * warps;
        }
      }
    }
  }
  L->ap = p;
}

// row pitch of the operator's D [q][ez][ey][ex]: a multiple of 16 bytes where the storage
// (54 reals an element) holds it
int hm_jac_pitch(const Lattice& L, int precision) {
  const int A = precision == HM_FP32 ? 4 : 2, p = (L.nx + A - 1) / A * A;
  return p <= 2 * L.nx ? p : L.nx;
}

namespace {
// raises a kernel's dynamic shared memory limit, once per device
template <typename K>
int raise_smem(K kern, std::atomic<uint64_t>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return HM_ERR_CUDA;
  if (dev < 0 || dev >= 64) return HM_ERR_UNSUPPORTED;
  if (!((done.load() >> dev) & 1u)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024) != cudaSuccess)
      return HM_ERR_CUDA;
    done.fetch_or(1ull << dev);
  }
  return HM_OK;
}
// the map of D [q][ez][ey][ex] with rows `pitch` apart; *tma = 0 where its storage has no
// 16-byte base or pitch
template <typename real>
int map_D(const Lattice& L, const void* D, int pitch, CUtensorMap* map, int* tma) {
  *tma = (reinterpret_cast<uintptr_t>(D) & 15u) == 0 && pitch * sizeof(real) % 16 == 0;
  if (!*tma) return HM_OK;
  auto encode = hm_tensor_map_encoder();
  if (encode == nullptr) return HM_ERR_CUDA;
  const cuuint64_t row = (cuuint64_t)pitch * sizeof(real);
  const cuuint64_t dims[4] = {(cuuint64_t)L.nx, (cuuint64_t)L.ny, (cuuint64_t)L.nz, 27};
  const cuuint64_t strides[3] = {row, row * L.ny, row * L.ny * L.nz};
  const cuuint32_t box[4] = {(cuuint32_t)box_columns<real>(L.ap.T1), (cuuint32_t)L.ap.T2, 1, 27};
  const cuuint32_t one[4] = {1, 1, 1, 1};
  return encode(map, sizeof(real) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                const_cast<void*>(D), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? HM_OK : HM_ERR_CUDA;
}
template <typename real, typename src, typename vec, int IN, int OUT>
int launch(const Lattice& L, const void* jac, int pitch, PassArgs<src, vec, OUT> a, void* stream) {
  auto kern = k_apply_tile<real, src, vec, IN, OUT>;
  static std::atomic<uint64_t> done{0};
  int rc = raise_smem(kern, done);
  if (rc) return rc;
  a.pitch = pitch;
  a.status = hm_status_word();
  CUtensorMap map{};
  if ((rc = map_D<real>(L, jac, pitch, &map, &a.tma))) return rc;
  kern<<<L.ap.t1 * L.ap.t2 * L.ap.t3, L.ap.threads, (size_t)ApplySmem<real, src>(L.ap).bytes,
         reinterpret_cast<cudaStream_t>(stream)>>>(map, L, static_cast<const real*>(jac), a);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}
template <typename real, typename src, typename vec, int IN, int OUT>
int launch(const Lattice& L, const void* jac, const PassArgs<src, vec, OUT>& a, void* stream) {
  return launch<real, src, vec, IN, OUT>(L, jac, hm_jac_pitch(L, sizeof(real) == 8 ? HM_FP64 : HM_FP32), a, stream);
}
template <typename real, typename T>
int apply_y(const Lattice& L, const void* jac, const uint8_t* ess, const T* x, T* y, bool clean,
            double* part, double* sc, unsigned* counter, double* fail, void* stream) {
  ApplyArgs<T, T> a{};
  a.ess = ess; a.x = x; a.y = y; a.part = part; a.fail = fail;
  a.sc = part != nullptr ? sc : nullptr;
  a.counter = counter;
  if (clean) return launch<real, T, T, IN_CLEAN, OUT_Y>(L, jac, a, stream);
  return launch<real, T, T, IN_ESS, OUT_Y>(L, jac, a, stream);
}
}  // namespace

int hm_launch_apply_A(const Lattice& L, void* jac, int precision, const uint8_t* ess,
                      const double* x, double* y, void* stream, double* fail) {
  if (precision == HM_FP32) return apply_y<float>(L, jac, ess, x, y, false, nullptr, nullptr, nullptr, fail, stream);
  return apply_y<double>(L, jac, ess, x, y, false, nullptr, nullptr, nullptr, fail, stream);
}

// with sc and counter the last block also takes the CG step's alpha; x must be zero on
// the Dirichlet nodes (the solves keep every search direction so)
int hm_launch_apply_A_dot(const Lattice& L, void* jac, int precision, const uint8_t* ess,
                          const double* x, double* y, double* part, void* stream, double* sc,
                          unsigned* counter) {
  double* const fail = sc != nullptr ? sc + SC_FAIL : nullptr;
  if (precision == HM_FP32) return apply_y<float>(L, jac, ess, x, y, true, part, sc, counter, fail, stream);
  return apply_y<double>(L, jac, ess, x, y, true, part, sc, counter, fail, stream);
}

int hm_launch_apply_A_clean(const Lattice& L, void* jac, const uint8_t* ess, const double* x,
                            double* y, void* stream) {
  return apply_y<double>(L, jac, ess, x, y, true, nullptr, nullptr, nullptr, nullptr, stream);
}

// y = D^-1 A x, x zero on the Dirichlet nodes: a step of the power iteration
int hm_launch_power(const Lattice& L, void* jac, const uint8_t* ess, const double* idiag, const double* x,
                    double* y, void* stream) {
  SmoothArgs<double, double> a{};
  a.ess = ess; a.x = x; a.y = y; a.c.idiag = idiag;
  return launch<double, double, double, IN_CLEAN, OUT_POWER>(L, jac, a, stream);
}

int hm_launch_apply_A32(const Lattice& L, void* jac32, const uint8_t* ess, const float* x,
                        float* y, bool clean, void* stream) {
  return apply_y<float>(L, jac32, ess, x, y, clean, nullptr, nullptr, nullptr, nullptr, stream);
}

// the FP32 operator on FP32 vectors (the inner solves of the mixed-precision PCG), x zero
// on the Dirichlet nodes
int hm_launch_apply_A32_dot(const Lattice& L, void* jac32, const uint8_t* ess, const float* x,
                            float* y, double* part, void* stream, double* sc, unsigned* counter) {
  return apply_y<float>(L, jac32, ess, x, y, true, part, sc, counter, sc != nullptr ? sc + SC_FAIL : nullptr, stream);
}

// A pass of the multigrid smoother: the arithmetic of its start / step / finish kernels.
// In the FP32 cycle in, x, r and dout are FP32; b, the update and z stay FP64.
template <typename T>
int hm_launch_cheb(const Lattice& L, void* jac, const uint8_t* ess, const HmCheb<T>& c, void* stream) {
  SmoothArgs<T, T> a{};
  a.ess = ess; a.x = c.in; a.fail = c.fail;
  a.c = {c.k, c.first, c.last, c.b, c.idiag, c.cheb, c.x, c.r, c.dout, c.z};
  if (c.beta != nullptr && (c.mode == CH_STEP1 || (c.mode == CH_NEXT && c.last == 2))) {
    a.part = c.beta->rz; a.sc = c.beta->sc; a.counter = c.beta->counter;
    a.rr = c.beta->rr; a.nrr = c.beta->n; a.flex = c.beta->flex;
    c.beta->done = 1;
  }
  switch (c.mode) {
    case CH_RESIDUAL: return launch<T, T, T, IN_CLEAN, OUT_R>(L, jac, a, stream);
    case CH_STEP1: return launch<T, T, T, IN_CLEAN, OUT_STEP1>(L, jac, a, stream);
    case CH_START: return launch<T, T, T, IN_CLEAN, OUT_START>(L, jac, a, stream);
    default: return launch<T, T, T, IN_CLEAN, OUT_NEXT>(L, jac, a, stream);
  }
}
template int hm_launch_cheb<double>(const Lattice&, void*, const uint8_t*, const HmCheb<double>&, void*);
template int hm_launch_cheb<float>(const Lattice&, void*, const uint8_t*, const HmCheb<float>&, void*);
int hm_launch_beta(const Lattice& L, const double* b, const double* z, const HmBeta& be, void* stream) {
  k_tile_beta<<<L.ap.t1 * L.ap.t2 * L.ap.t3, L.ap.threads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(L, b, z, be);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}

// The assembled vectors from the fields.  D: storage of at least 27 ne doubles (54 ne for
// its 16-byte pitch where nx is odd), work_reals of them, 27 ne a vector at least; outs:
// ADJOINT, STATE, PARAMETER (NULL: skip).  With skip nonzero on the device nothing is done.
int hm_launch_vectors(const Lattice& L, const double* u, const double* m, const double* p,
                      const double* mhat, double f, const uint8_t* zero_ess, double* const outs[3],
                      double* D, int64_t work_reals, uint32_t* status, const uint32_t* skip, void* stream) {
  // The passes write nodes while other tiles, and the other vectors' passes, still read u and
  // p: an output that overlaps either takes the element route.
  auto overlaps = [&](const double* out, const double* x) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(out), b = reinterpret_cast<uintptr_t>(x);
    const uintptr_t bytes = sizeof(double) * (uintptr_t)L.ndof;
    return a < b + bytes && b < a + bytes;
  };
  // And one or two vectors on a small mesh, where the passes are latency -- k_points_D, then
  // layers in series: 11 to 13 us whatever the size, against 7 to 10 for one vector by the
  // element route up to 14^3 (10.1 against 11.1-12.5; 16^3 12.0 against 11.1-12.3, 20^3 17.0
  // against 11.7-13) and 10 to 12 for two up to 12^3 (12.0 against 12.6; 14^3 13.5 against
  // 12.9); three take 13.3 either way at 8^3.  Not on a slab: the routes sum in other orders.
  const int count = (outs[0] != nullptr) + (outs[1] != nullptr) + (outs[2] != nullptr);
  bool element = !L.slab && ((count == 1 && L.ne <= 2744) || (count == 2 && L.ne <= 1728));
  for (int i = 0; i < 3; ++i)
    if (outs[i] && (overlaps(outs[i], u) || overlaps(outs[i], p))) element = true;
  if (element) return hm_launch_elem_vectors(L, u, m, p, mhat, f, zero_ess, outs, D, status, skip, stream);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int pitch = hm_jac_pitch(L, HM_FP64);
  if (27 * (int64_t)pitch * L.ny * L.nz > work_reals) pitch = L.nx;
  k_points_D<<<(int)((L.ne + 127) / 128), 128, 0, s>>>(L, pitch, u, m, p, mhat, D, status, skip);
  static std::atomic<uint64_t> done{0};
  int rc = raise_smem(k_vectors, done);
  if (rc) return rc;
  CUtensorMap map{};
  VecArgs v{};
  v.u = u; v.p = p; v.grad = outs[2]; v.skip = skip;
  for (int i = 0; i < 2; ++i) {
    VecPart& a = v.a[i];
    a.ess = zero_ess; a.x = i == 0 ? u : p; a.y = outs[i];
    a.f = i == 0 && mhat == nullptr ? f : 0.0;
    const double h[3] = {L.hx, L.hy, L.hz};
    for (int d = 0; d < 3; ++d) {
      a.phi[d][0] = h[d] * (2.0 / 3.0); a.phi[d][1] = h[d] / 6.0; a.phi[d][2] = h[d] / 3.0;
    }
    a.pitch = pitch;
    a.status = hm_status_word();
    a.caller = status;
    a.sx = 1.0 / (0.6 * L.hx * L.hx);
    a.ry = (L.hx * L.hx) / (L.hy * L.hy);
    a.rz = (L.hx * L.hx) / (L.hz * L.hz);
    if ((rc = map_D<double>(L, D, pitch, &map, &a.tma))) return rc;
  }
  for (int i = 0; i < 3; ++i)
    if (outs[i]) v.which[v.count++] = i;
  const int bytes = ApplySmem<double, double>(L.ap).bytes, grad = GradSmem(L.ap).bytes;
  const bool applies = outs[0] || outs[1];
  k_vectors<<<L.ap.t1 * L.ap.t2 * L.ap.t3 * v.count, L.ap.threads,
              (size_t)(!outs[2] || (applies && bytes > grad) ? bytes : grad), s>>>(map, L, D, v);
  return cudaGetLastError() == cudaSuccess ? HM_OK : HM_ERR_CUDA;
}
