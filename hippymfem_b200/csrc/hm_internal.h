// Launchers shared between the translation units of libhippymfem_b200.
#pragma once

#include <cstdint>

#include "../../include/hippymfem_b200.h"

namespace hm {
struct Lattice;
}

// the geometry behind a lattice handle
const hm::Lattice* hm_lattice_geometry(const hm_lattice* h);
// the device address of the library's status word (hm_device_status)
uint32_t* hm_status_word();
// row pitch of the matrix-free operator's D [q][ez][ey][ex]
int hm_jac_pitch(const hm::Lattice& L, int precision);
// the tiling of the matrix-free apply for the lattice's sizes
void hm_plan_apply(hm::Lattice* L);

int hm_launch_pattern(const hm::Lattice& L, int32_t* indptr, int32_t* indices, int32_t* slot,
                      void* stream);
int hm_launch_tpos(const hm::Lattice& L, const int32_t* indptr, int32_t* tpos, void* stream);
int hm_launch_quad(const hm::Lattice& L, const double* u, const double* m, const double* p,
                   int precision, void* quad, uint32_t* status, void* stream,
                   const double* mhat = nullptr);
int hm_launch_assemble(const hm::Lattice& L, const void* quad, int precision,
                       const int32_t* indptr, const uint8_t* ess, double f, double* vA,
                       double* vC, double* vWum, double* vWmm, double* vs, double* vp,
                       double* va, int zero_ess, void* stream);
int hm_launch_jacobian_prepare(const hm::Lattice& L, const void* quad, int quad_precision,
                               void* jac, int precision, void* stream);
int hm_launch_apply_A(const hm::Lattice& L, void* jac, int precision, const uint8_t* ess,
                      const double* x, double* y, void* stream, double* fail = nullptr);
int hm_launch_diag_A(const hm::Lattice& L, const void* quad, int precision,
                     const uint8_t* ess, double* diag, void* stream);
int hm_launch_apply_A_dot(const hm::Lattice& L, void* jac, int precision, const uint8_t* ess,
                          const double* x, double* y, double* part, void* stream,
                          double* sc = nullptr, unsigned* counter = nullptr);
int hm_launch_apply_A32_dot(const hm::Lattice& L, void* jac32, const uint8_t* ess, const float* x,
                            float* y, double* part, void* stream, double* sc = nullptr,
                            unsigned* counter = nullptr);
// y = A x for an x that is zero on the Dirichlet nodes (FP64 operator)
int hm_launch_apply_A_clean(const hm::Lattice& L, void* jac, const uint8_t* ess, const double* x,
                            double* y, void* stream);
// the assembled vectors from the fields (hm_apply.cu)
int hm_launch_vectors(const hm::Lattice& L, const double* u, const double* m, const double* p,
                      const double* mhat, double f, const uint8_t* zero_ess, double* const outs[3],
                      double* D, int64_t work_reals, uint32_t* status, const uint32_t* skip, void* stream);
// the same by the element route, whose outputs may overlap the fields (hm_lattice.cu)
int hm_launch_elem_vectors(const hm::Lattice& L, const double* u, const double* m, const double* p,
                           const double* mhat, double f, const uint8_t* zero_ess, double* const outs[3],
                           double* work, uint32_t* status, const uint32_t* skip, void* stream);
// x = b on the Dirichlet nodes
int hm_launch_ess_take_b(const hm::Lattice& L, const uint8_t* ess, const double* b, double* x,
                         void* stream);
// the right-hand side and solution buffers a solve plan was created with
int hm_plan_buffers(const hm_pcg_plan* plan, double** b, double** x);
// the FP32 operator (jac32: the points' D in FP32) on FP32 vectors; clean: x zero on the Dirichlet nodes
int hm_launch_apply_A32(const hm::Lattice& L, void* jac32, const uint8_t* ess, const float* x,
                        float* y, bool clean, void* stream);
// Inside the MG-PCG: r.z and the step's beta, taken by the cycle's last operator pass
// (done set) where it can: rz room for its partials, rr the n partials of r.r, then those of
// r.z_old with flex
struct HmBeta {
  double* rz;
  const double* rr;
  unsigned n;
  int flex;
  double* sc;
  unsigned* counter;
  int done;
};
// the same on its own
int hm_launch_beta(const hm::Lattice& L, const double* b, const double* z, const HmBeta& be, void* stream);
// fail: the solve's SC_FAIL, set where a fused level-0 pass gives up a wait
int hm_mg_vcycle(hm_mg* mg, const double* r, double* z, void* stream, double* fail, HmBeta* beta = nullptr);
// One operator pass of the level-0 Chebyshev-Jacobi smoother (hm_apply.cu), every vector
// zero on the Dirichlet nodes, T the cycle's precision:
//   CH_RESIDUAL  r = b - A in                     (degree 1: in = x = the first direction)
//   CH_STEP1     z = in + (b - A in) idiag / theta, z != in
//   CH_START     r = b - A in, dout = r idiag / theta
//   CH_NEXT      step k: r -= A in (first: r = b - A in), x += in (first: x = in),
//                dout = c1_k in + c2_k r idiag; last = 1: no dout; last = 2: z = x + dout,
//                nothing else stored
// With beta (CH_STEP1, or CH_NEXT with last = 2) the pass also takes b.z and the CG
// step's beta.
enum HmChebMode { CH_RESIDUAL = 0, CH_STEP1 = 1, CH_START = 2, CH_NEXT = 3 };
template <typename T>
struct HmCheb {
  int mode, k, first, last;
  const double* b;
  const double* idiag;
  const double* cheb;
  const T* in;
  T* x;
  T* r;
  T* dout;
  double* z;
  HmBeta* beta;
  double* fail;             // the solve's SC_FAIL (NULL: none)
};
template <typename T>
int hm_launch_cheb(const hm::Lattice& L, void* jac, const uint8_t* ess, const HmCheb<T>& c, void* stream);
// y = D^-1 A x, x zero on the Dirichlet nodes (a step of the set-up's power iteration)
int hm_launch_power(const hm::Lattice& L, void* jac, const uint8_t* ess, const double* idiag, const double* x,
                    double* y, void* stream);
// Inside the MG-PCG: where the level-0 smoother's first direction d = r idiag / theta is
// wanted (d64 or d32; both null: nowhere), formed by the kernel that forms r
struct HmFirstDir {
  const double* idiag;
  const double* cheb;
  double* d64;
  float* d32;
};
HmFirstDir hm_mg_first_dir(const hm_mg* mg);
