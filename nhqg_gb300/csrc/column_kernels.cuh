// Column kernels: everything that acts on one horizontal mode's vertical
// column.  Each CTA owns TM consecutive compact modes and stages their
// columns (all levels) in shared memory as tiles [level][TM].
//
// Reference operations (nhqg/solver.py):
//   Chebyshev <-> CGL nodal transforms V, V^-1           :45-52
//   Galerkin stencil S and its exact left inverse pinv   :65-72 (grid.py:497-506, 322-342)
//   d/dZ on Chebyshev coefficients G_Z                    grid.py:148-169
//   explicit-RHS assembly                                 :541-549
//   implicit tendency                                     :615-641
//   implicit solve (block elimination)                    :691-738
//   stage combinations of ARS(2,2,2) / SBP2-PC            :1023-1048, :1205-1217
//   finalize + sanitize                                   :993-999, :128-146
// pinv_w(proj_w(x)) == pinv_w(x) because pinv reads only the first Nz-1
// Chebyshev coefficients and the tau projection rewrites only the last two,
// so the tau projections that feed a pinv are not applied.
//
// The kernels are templates on TM, instantiated by column_tm2.cu, _tm4.cu and
// _tm8.cu; column_modes() picks TM by the depth and the number of modes.
#pragma once
#include <algorithm>
#include <type_traits>

#include "column.cuh"
#include "engine.h"

namespace nhqg {
namespace colk {

using col::NT;

struct VK {
  int P, G, N, M, Mr, Mc, K, Nx, Nk;
  bool mixed;                 // open-top (Neumann) w basis
  const double *wa, *wb;      // mixed stencil coefficients
  col::Dct dct;
  const double *kx, *inv_denom, *inv_aq, *inv_at, *drq, *drw, *drt;
  double beta, Ra, gdt;
};

inline VK make_vk(const Params& p, const Tables& t) {
  VK k;
  k.P = p.d.P; k.G = p.d.G; k.N = p.d.Nz; k.M = p.d.M; k.Mr = p.d.Mr; k.Mc = p.d.Mc;
  k.K = p.d.K; k.Nx = p.d.Nx; k.Nk = p.d.Nk;
  k.mixed = t.wst_a != nullptr;
  k.wa = t.wst_a; k.wb = t.wst_b;
  k.dct = make_dct(p, t);
  k.kx = t.kx; k.inv_denom = t.inv_denom; k.inv_aq = t.inv_aq; k.inv_at = t.inv_at;
  k.drq = t.drq; k.drw = t.drw; k.drt = t.drt;
  k.beta = p.beta; k.Ra = p.Ra_sigma; k.gdt = p.gamma_imex * p.dt;
  return k;
}

template <int TM, typename C>
__device__ __forceinline__ void tstencil_w(const VK& k, C* c, const C* x) {
  using Cl = col::Cols<TM>;
  if (!k.mixed) Cl::tstencil_dir(c, x, k.P, k.G);
  else Cl::tstencil_mixed(c, x, k.P, k.G, k.wa, k.wb);
}
template <int TM, typename C>
__device__ __forceinline__ void tpinv_w(const VK& k, C* x, const C* c) {
  using Cl = col::Cols<TM>;
  if (!k.mixed) Cl::tpinv_dir(x, c, k.G);
  else Cl::tpinv_mixed(x, c, k.G, k.wa, k.wb);
}

// =========================================================== forward: to nodal
// DCT of the FP64 tile src (ready) to nodal values in the precision of CO,
// stored to out; spare is a free FP64 tile used as scratch.
template <int TM, typename CO>
__device__ __forceinline__ void to_nodal(const VK& k, const col::DctSharedT<CO>& ds,
                                         const double2* src, double2* spare, CO* out, int m0) {
  using Cl = col::Cols<TM>;
  if constexpr (sizeof(CO) == sizeof(double2)) {
    Cl::tdct(spare, src, k.dct, ds, false, k.P);
    __syncthreads();
    Cl::tstore(spare, out, k.P, m0, k.M);
  } else {
    float2* fs = reinterpret_cast<float2*>(spare);
    float2* fo = fs + k.P * TM;
    Cl::tcvt(fs, src, k.P);
    __syncthreads();
    Cl::tdct(fo, fs, k.dct, ds, false, k.P);
    __syncthreads();
    Cl::tstore(fo, out, k.P, m0, k.M);
  }
}

// CO = double2: plain FP64 path; CO = float2: the mixed-precision path keeps
// the Galerkin stencils in FP64 and runs the DCT in FP32.
template <int TM, typename CO>
__global__ void __launch_bounds__(NT) k_vfwd(VK k, const double2* q, const double2* w,
                                             const double2* th, CO* qn, CO* wn, CO* tn) {
  using Cl = col::Cols<TM>;
  extern __shared__ double2 sm[];
  double2* b0 = sm;
  double2* b1 = sm + k.P * TM;
  const col::DctSharedT<CO> ds = Cl::template dct_shared<CO>(k.dct, sm + 2 * k.P * TM);
  after_previous();
  const int m0 = blockIdx.x * TM;
  if (q) {
    Cl::tload(b0, q, k.P, m0, k.M);
    __syncthreads();
    to_nodal<TM>(k, ds, b0, b1, qn, m0);
    __syncthreads();
  }
  if (w) {
    Cl::tload(b0, w, k.G, m0, k.M);
    __syncthreads();
    tstencil_w<TM>(k, b1, b0);
    __syncthreads();
    to_nodal<TM>(k, ds, b1, b0, wn, m0);
    __syncthreads();
  }
  if (th) {
    Cl::tload(b0, th, k.G, m0, k.M);
    __syncthreads();
    Cl::tstencil_dir(b1, b0, k.P, k.G);
    __syncthreads();
    to_nodal<TM>(k, ds, b1, b0, tn, m0);
  }
}

// form of the explicit operand A that k_vback reads
enum AKind {
  AK_F64 = 0,       // FP64 nodal values (plain path)
  AK_F32_NODAL = 1, // FP32 nodal values, inverse DCT in FP32
  AK_F32_COEF = 2,  // FP32 explicit tendencies from the tensor-core inverse:
                    // E_q (Chebyshev), E_w and E_theta (Galerkin, pinv applied)
};

// Chebyshev coefficients (FP64 tile out) of the explicit operand A, read in
// the form AK; tmp is a free tile.
template <int TM, int AK, typename DS, typename C>
__device__ __forceinline__ void a_to_coef(const VK& k, const DS& ds, const double2* Ad,
                                          const float2* Af, C* tmp, C* out, int m0) {
  using Cl = col::Cols<TM>;
  if constexpr (AK == AK_F32_COEF) {
    Cl::tloadp(out, Af, k.P, m0, k.M);
  } else if constexpr (AK == AK_F64) {
    Cl::tload(tmp, Ad, k.P, m0, k.M);
    __syncthreads();
    Cl::tdct(out, tmp, k.dct, ds, true, k.P);
  } else {
    float2* fi = reinterpret_cast<float2*>(tmp);
    float2* fo = fi + k.P * TM;
    Cl::tload(fi, Af, k.P, m0, k.M);
    __syncthreads();
    Cl::tdct(fo, fi, k.dct, ds, true, k.P);
    __syncthreads();
    Cl::tcvt(out, fo, k.P);
  }
}

// =========================================================== back + stage + solve-pre
// Tiles of type C: double2, or cdfl (double-float, the mixed path with the
// tensor-core inverse, AK_F32_COEF) -- fields in global memory stay FP64.
template <int TM, int MODE, int AK, typename C = double2>
__global__ void __launch_bounds__(NT) k_vback(VK k, VArgs a) {
  using Cl = col::Cols<TM>;
  static_assert(std::is_same<C, double2>::value || AK == AK_F32_COEF,
                "double-float tiles read the explicit operand as coefficients");
  using T = typename col::Prec<C>::T;
  using Pr = col::Prec<C>;
  extern __shared__ double2 sm_raw[];
  C* sm = reinterpret_cast<C*>(sm_raw);
  const int PT = k.P * TM;
  C *b0 = sm, *b1 = sm + PT, *b2 = sm + 2 * PT, *b3 = sm + 3 * PT, *b4 = sm + 4 * PT;
  using CA = typename std::conditional<AK == AK_F32_NODAL, float2, double2>::type;
  col::DctSharedT<CA> ds{};
  if constexpr (AK != AK_F32_COEF) ds = Cl::template dct_shared<CA>(k.dct, sm_raw + 5 * PT, b2);
  after_previous();
  const int m0 = blockIdx.x * TM;
  const int P = k.P, G = k.G, M = k.M;
  const size_t Ms = (size_t)M;
  const T alpha = Pr::s(a.alpha), cE1 = Pr::s(a.c_E1), cE2 = Pr::s(a.c_E2);
  const T omega = Pr::s(a.omega), gdt = Pr::s(k.gdt), Ra = Pr::s(k.Ra);
  // L2 prefetch of the CTA's columns of a field (the line holding modes m0,
  // m0 + 1 at every level), one field group ahead of the phase that reads it,
  // so that the phase's loads find L2 instead of waiting on DRAM
  auto pf = [&](const void* f, int nlev, size_t esize) {
    if (f == nullptr) return;
    const char* base = static_cast<const char*>(f) + (size_t)m0 * esize;
    for (int l = threadIdx.x; l < nlev; l += blockDim.x)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(base + (size_t)l * Ms * esize));
  };
  if constexpr (MODE == VB_STAGE2) {
    pf(a.w1, G, 16); pf(a.q0, P, 16); pf(a.E1q, P, 16); pf(a.q1, P, 16);
  } else if constexpr (MODE == VB_STAGE1) {
    pf(a.q0, P, 16); pf(AK == AK_F32_COEF ? (const void*)a.Awf : (const void*)nullptr, G, 8);
  }

  // ------------------------------------------------------------- q
  if (MODE != VB_SOLVE) {
    a_to_coef<TM, AK>(k, ds, a.Aq, a.Aqf, b0, b1, m0);
    __syncthreads();
    // E_q = -Aq - i beta kx psi, psi = -inv_denom * q_state
    const double2* qs = (MODE == VB_STAGE2) ? a.q1 : a.q0;
    for (int i = threadIdx.x; i < PT; i += blockDim.x) {
      const int l = i / TM, m = (m0 + i % TM);
      if (m >= M) continue;
      C e = (AK == AK_F32_COEF) ? b1[i] : col::gneg(b1[i]);
      if (k.beta != 0.0) {
        const T sb = Pr::s(k.beta * k.kx[m] * k.inv_denom[m]);
        const C qv = Pr::in(qs[(size_t)l * Ms + m]);
        e = gmk<C>(fma(-sb, qv.y, e.x), fma(sb, qv.x, e.y));
      }
      if (a.Cq) e = gadd(e, Pr::in(a.Cq[(size_t)l * Ms + m]));  // learned closure
      b1[i] = e;
    }
    __syncthreads();
    if (MODE == VB_RHS) {
      Cl::tstorep(b1, a.Eq, P, m0, M);
    } else if (MODE == VB_STAGE1) {
      Cl::tstorep(b1, a.E1q, P, m0, M);
      for (int i = threadIdx.x; i < PT; i += blockDim.x) {
        const int l = i / TM, m = (m0 + i % TM);
        if (m < M) b1[i] = col::gaxpy(alpha, b1[i], Pr::in(a.q0[(size_t)l * Ms + m]));
      }
    } else {  // STAGE2: I_q = G_Z S_w w1
      Cl::tloadp(b2, a.w1, G, m0, M);
      __syncthreads();
      tstencil_w<TM>(k, b3, b2);
      __syncthreads();
      Cl::tgz(b2, b3, k.N);
      __syncthreads();
      for (int i = threadIdx.x; i < PT; i += blockDim.x) {
        const int l = i / TM, m = (m0 + i % TM);
        if (m >= M) continue;
        const size_t g = (size_t)l * Ms + m;
        C r = Pr::in(a.q0[g]);
        r = col::gaxpy(cE1, Pr::in(a.E1q[g]), r);
        r = col::gaxpy(cE2, b1[i], r);
        r = col::gaxpy(omega, b2[i], r);
        r = col::gaxpy((-omega) * Pr::s(k.drq[m]), Pr::in(a.q1[g]), r);
        b1[i] = r;
      }
    }
    __syncthreads();
  } else {
    Cl::tloadp(b1, a.q0, P, m0, M);  // R_q given
    __syncthreads();
  }
  if (MODE != VB_RHS) {
    Cl::tstorep(b1, a.Rq, P, m0, M);
    // temp = R_q / alpha_q ; d_gal = pinv_w(inv_denom * G_Z temp)
    for (int i = threadIdx.x; i < PT; i += blockDim.x) {
      const int m = (m0 + i % TM);
      b2[i] = (m < M) ? gscale(b1[i], Pr::s(k.inv_aq[m])) : col::gzero<C>();
    }
    __syncthreads();
    Cl::tgz(b3, b2, k.N);
    __syncthreads();
    for (int i = threadIdx.x; i < PT; i += blockDim.x) {
      const int m = (m0 + i % TM);
      b3[i] = (m < M) ? gscale(b3[i], Pr::s(k.inv_denom[m])) : col::gzero<C>();
    }
    __syncthreads();
    tpinv_w<TM>(k, b4, b3);
    __syncthreads();
  }

  // ------------------------------------------------------------- w
  if constexpr (MODE == VB_STAGE2) {
    if constexpr (AK == AK_F32_COEF) pf(a.Awf, G, 8);
    pf(a.t1, G, 16); pf(a.w0, G, 16); pf(a.E1w, G, 16);
  } else if constexpr (MODE == VB_STAGE1) {
    pf(a.w0, G, 16);
    if constexpr (AK == AK_F32_COEF) pf(a.Atf, G, 8);
  }
  if (MODE != VB_SOLVE) {
    if constexpr (AK == AK_F32_COEF) {  // E_w in the Galerkin basis
      Cl::tloadp(b2, a.Awf, G, m0, M);
    } else {
      a_to_coef<TM, AK>(k, ds, a.Aw, a.Awf, b0, b1, m0);
      __syncthreads();
      for (int i = threadIdx.x; i < PT; i += blockDim.x) b1[i] = col::gneg(b1[i]);
      __syncthreads();
      tpinv_w<TM>(k, b2, b1);
    }
    __syncthreads();
    if (MODE == VB_RHS) {
      Cl::tstorep(b2, a.Ew, G, m0, M);
    } else if (MODE == VB_STAGE1) {
      Cl::tstorep(b2, a.E1w, G, m0, M);
      for (int i = threadIdx.x; i < G * TM; i += blockDim.x) {
        const int l = i / TM, m = (m0 + i % TM);
        if (m < M) b2[i] = col::gaxpy(alpha, b2[i], Pr::in(a.w0[(size_t)l * Ms + m]));
      }
    } else {  // I_w = pinv_w(inv_denom G_Z q1 + Ra S_dir t1)
      Cl::tloadp(b0, a.q1, P, m0, M);
      __syncthreads();
      Cl::tgz(b1, b0, k.N);
      __syncthreads();
      Cl::tloadp(b0, a.t1, G, m0, M);
      __syncthreads();
      Cl::tstencil_dir(b3, b0, P, G);
      __syncthreads();
      for (int i = threadIdx.x; i < PT; i += blockDim.x) {
        const int m = (m0 + i % TM);
        b1[i] = (m < M) ? col::gaxpy(Ra, b3[i], gscale(b1[i], Pr::s(k.inv_denom[m]))) : col::gzero<C>();
      }
      __syncthreads();
      tpinv_w<TM>(k, b0, b1);
      __syncthreads();
      for (int i = threadIdx.x; i < G * TM; i += blockDim.x) {
        const int l = i / TM, m = (m0 + i % TM);
        if (m >= M) continue;
        const size_t g = (size_t)l * Ms + m;
        C r = Pr::in(a.w0[g]);
        r = col::gaxpy(cE1, Pr::in(a.E1w[g]), r);
        r = col::gaxpy(cE2, b2[i], r);
        r = col::gaxpy(omega, b0[i], r);
        r = col::gaxpy((-omega) * Pr::s(k.drw[m]), Pr::in(a.w1[g]), r);
        b2[i] = r;
      }
    }
    __syncthreads();
  } else {
    Cl::tloadp(b2, a.w0, G, m0, M);  // R_w given
    __syncthreads();
  }
  if (MODE != VB_RHS) {
    for (int i = threadIdx.x; i < G * TM; i += blockDim.x) b4[i] = col::gaxpy(gdt, b4[i], b2[i]);
    __syncthreads();
  }

  // ------------------------------------------------------------- theta
  if constexpr (MODE == VB_STAGE2) {
    if constexpr (AK == AK_F32_COEF) pf(a.Atf, G, 8);
    pf(a.t0, G, 16); pf(a.E1t, G, 16); pf(a.t1p, G, 16);
  } else if constexpr (MODE == VB_STAGE1) {
    pf(a.t0, G, 16);
  }
  if (MODE != VB_SOLVE) {
    if constexpr (AK == AK_F64) {
      Cl::tload(b0, a.At, P, m0, M);
      __syncthreads();
      if (a.dtb_nodal != nullptr) {  // legacy evolve_mean: + (dTheta/dZ)_nodal * w_nodal
        for (int i = threadIdx.x; i < PT; i += blockDim.x) {
          const int l = i / TM, m = (m0 + i % TM);
          if (m < M) b0[i] = caxpy(a.dtb_nodal[l], a.Wn[(size_t)l * Ms + m], b0[i]);
        }
        __syncthreads();
      }
      Cl::tdct(b1, b0, k.dct, ds, true, P);
    } else if constexpr (AK == AK_F32_NODAL) {  // the mixed path has no legacy evolve_mean term
      a_to_coef<TM, AK>(k, ds, nullptr, a.Atf, b0, b1, m0);
    }
    if constexpr (AK == AK_F32_COEF) {  // E_theta in the Galerkin basis
      Cl::tloadp(b2, a.Atf, G, m0, M);
    } else {
      __syncthreads();
      for (int i = threadIdx.x; i < PT; i += blockDim.x) b1[i] = col::gneg(b1[i]);
      __syncthreads();
      Cl::tpinv_dir(b2, b1, G);
    }
    __syncthreads();
    if (MODE == VB_RHS) {
      Cl::tstorep(b2, a.Et, G, m0, M);
    } else if (MODE == VB_STAGE1) {
      Cl::tstorep(b2, a.E1t, G, m0, M);
      for (int i = threadIdx.x; i < G * TM; i += blockDim.x) {
        const int l = i / TM, m = (m0 + i % TM);
        if (m < M) b2[i] = col::gaxpy(alpha, b2[i], Pr::in(a.t0[(size_t)l * Ms + m]));
      }
    } else {  // I_t = w1 (shared basis) or pinv_dir(S_w w1)
      Cl::tloadp(b0, a.w1, G, m0, M);
      __syncthreads();
      if (k.mixed) {
        tstencil_w<TM>(k, b1, b0);
        __syncthreads();
        Cl::tpinv_dir(b0, b1, G);
        __syncthreads();
      }
      const T iac = Pr::s(a.inv_alpha_c);
      for (int i = threadIdx.x; i < G * TM; i += blockDim.x) {
        const int l = i / TM, m = (m0 + i % TM);
        if (m >= M) continue;
        const size_t g = (size_t)l * Ms + m;
        C r = Pr::in(a.t0[g]);
        r = col::gaxpy(cE1, Pr::in(a.E1t[g]), r);
        r = col::gaxpy(cE2, b2[i], r);
        r = col::gaxpy(omega, b0[i], r);
        const C t1v = Pr::in(a.t1[g]);
        r = col::gaxpy((-omega) * Pr::s(k.drt[m]), t1v, r);
        if (a.inv_alpha_c != 0.0) {
          const C c = gscale(gsub(t1v, Pr::in(a.t1p[g])), iac);
          r = col::gaxpy(omega, c, r);
        }
        b2[i] = r;
      }
    }
    __syncthreads();
  } else {
    Cl::tloadp(b2, a.t0, G, m0, M);  // R_th given
    __syncthreads();
  }
  if (MODE != VB_RHS) {
    Cl::tstorep(b2, a.Rt, G, m0, M);
    for (int i = threadIdx.x; i < G * TM; i += blockDim.x) {
      const int m = (m0 + i % TM);
      b0[i] = (m < M) ? gscale(b2[i], Pr::s(k.inv_at[m])) : col::gzero<C>();
    }
    __syncthreads();
    if (k.mixed) {  // theta basis -> w basis
      Cl::tstencil_dir(b1, b0, P, G);
      __syncthreads();
      tpinv_w<TM>(k, b0, b1);
      __syncthreads();
    }
    const T c = Pr::s(k.gdt * k.Ra);
    for (int i = threadIdx.x; i < G * TM; i += blockDim.x) b4[i] = col::gaxpy(c, b0[i], b4[i]);
    __syncthreads();
    Cl::tstorep(b4, a.rhs_w, G, m0, M);
  }
}

// =========================================================== back-substitution
template <int TM, typename C = double2>
__global__ void __launch_bounds__(NT) k_vpost(VK k, const double2* Rq, const double2* Rt,
                                              const double2* wn, double2* qo, double2* to,
                                              bool zero_mean) {
  after_previous();
  using Cl = col::Cols<TM>;
  using Pr = col::Prec<C>;
  extern __shared__ double2 sm_raw[];
  C* sm = reinterpret_cast<C*>(sm_raw);
  const int PT = k.P * TM;
  C *b0 = sm, *b1 = sm + PT, *b2 = sm + 2 * PT;
  const int m0 = blockIdx.x * TM;
  const int M = k.M;
  const typename Pr::T gdt = Pr::s(k.gdt);
  Cl::tprefetch(Rq, k.P, m0, M, sizeof(double2));
  Cl::tprefetch(Rt, k.G, m0, M, sizeof(double2));
  Cl::tloadp(b0, wn, k.G, m0, M);
  __syncthreads();
  tstencil_w<TM>(k, b1, b0);  // w Chebyshev coefficients
  __syncthreads();
  Cl::tgz(b2, b1, k.N);
  __syncthreads();
  for (int i = threadIdx.x; i < PT; i += blockDim.x) {
    const int l = i / TM, m = (m0 + i % TM);
    if (m >= M) continue;
    const size_t g = (size_t)l * M + m;
    qo[g] = (zero_mean && m == 0) ? czero()
                                  : Pr::out(gscale(col::gaxpy(gdt, b2[i], Pr::in(Rq[g])), Pr::s(k.inv_aq[m])));
  }
  if (k.mixed) {  // w basis -> theta basis
    __syncthreads();
    Cl::tpinv_dir(b0, b1, k.G);
    __syncthreads();
  }
  for (int i = threadIdx.x; i < k.G * TM; i += blockDim.x) {
    const int l = i / TM, m = (m0 + i % TM);
    if (m >= M) continue;
    const size_t g = (size_t)l * M + m;
    to[g] = (zero_mean && m == 0) ? czero()
                                  : Pr::out(gscale(col::gaxpy(gdt, b0[i], Pr::in(Rt[g])), Pr::s(k.inv_at[m])));
  }
}

// =========================================================== implicit tendency
template <int TM>
__global__ void __launch_bounds__(NT) k_itend(VK k, const double2* q, const double2* w,
                                              const double2* th, double2* Iq, double2* Iw,
                                              double2* It) {
  after_previous();
  using Cl = col::Cols<TM>;
  extern __shared__ double2 sm[];
  const int PT = k.P * TM;
  double2 *b0 = sm, *b1 = sm + PT, *b2 = sm + 2 * PT, *b3 = sm + 3 * PT;
  const int m0 = blockIdx.x * TM;
  const int M = k.M;
  Cl::tload(b0, w, k.G, m0, M);
  __syncthreads();
  tstencil_w<TM>(k, b1, b0);
  __syncthreads();
  Cl::tgz(b2, b1, k.N);
  __syncthreads();
  Cl::tstore(b2, Iq, k.P, m0, M);
  if (k.mixed) {
    Cl::tpinv_dir(b3, b1, k.G);
    __syncthreads();
    Cl::tstore(b3, It, k.G, m0, M);
  } else {
    Cl::tstore(b0, It, k.G, m0, M);
  }
  __syncthreads();
  Cl::tload(b0, q, k.P, m0, M);
  __syncthreads();
  Cl::tgz(b1, b0, k.N);
  Cl::tload(b2, th, k.G, m0, M);
  __syncthreads();
  Cl::tstencil_dir(b3, b2, k.P, k.G);
  __syncthreads();
  for (int i = threadIdx.x; i < PT; i += blockDim.x) {
    const int m = (m0 + i % TM);
    b1[i] = (m < M) ? caxpy(k.Ra, b3[i], cscale(b1[i], k.inv_denom[m])) : czero();
  }
  __syncthreads();
  tpinv_w<TM>(k, b0, b1);
  __syncthreads();
  Cl::tstore(b0, Iw, k.G, m0, M);
}

// dynamic shared memory of a column kernel: nbuf FP64 tiles plus the DCT
// work area in FP64 or (f32_dct) FP32
template <int TM>
inline size_t vsmem(const Params& p, int nbuf, bool dct = false, bool f32_dct = false, bool own_work = true) {
  size_t b = (size_t)nbuf * p.d.P * TM * sizeof(double2);
  if (dct) b += col::Cols<TM>::dct_smem_bytes(make_dct(p, Tables{}), f32_dct, own_work);
  return b;
}
template <int TM>
inline int vgrid(const Params& p) { return (p.d.M + TM - 1) / TM; }

template <int TM, typename CO>
cudaError_t vfwd_t(const Params& p, const Tables& t, const double2* q, const double2* w,
                   const double2* th, CO* qn, CO* wn, CO* tn, cudaStream_t st) {
  VK k = make_vk(p, t);
  const size_t sm = vsmem<TM>(p, 2, true, sizeof(CO) == sizeof(float2));
  launch_after(k_vfwd<TM, CO>, vgrid<TM>(p), NT, sm, st, k, q, w, th, qn, wn, tn);
  return cudaGetLastError();
}

template <int TM, int MODE, int AK, typename C = double2>
void vback_t(const VK& k, const VArgs& a, size_t sm, int grid, cudaStream_t st) {
  launch_after(k_vback<TM, MODE, AK, C>, grid, NT, sm, st, k, a);
}
template <int TM, int MODE>
void vback_ak(int ak, const VK& k, const VArgs& a, size_t sm, int grid, cudaStream_t st) {
  if (ak == AK_F64) vback_t<TM, MODE, AK_F64>(k, a, sm, grid, st);
  else if (ak == AK_F32_NODAL) vback_t<TM, MODE, AK_F32_NODAL>(k, a, sm, grid, st);
  else if (a.df) vback_t<TM, MODE, AK_F32_COEF, cdfl>(k, a, sm, grid, st);
  else vback_t<TM, MODE, AK_F32_COEF>(k, a, sm, grid, st);
}

}  // namespace colk

template <int TM>
cudaError_t ColumnOps<TM>::vfwd(const Params& p, const Tables& t, const double2* q, const double2* w,
                                const double2* th, double2* qn, double2* wn, double2* tn, cudaStream_t st) {
  return colk::vfwd_t<TM>(p, t, q, w, th, qn, wn, tn, st);
}

template <int TM>
cudaError_t ColumnOps<TM>::vfwd_f32(const Params& p, const Tables& t, const double2* q, const double2* w,
                                    const double2* th, float2* qn, float2* wn, float2* tn, cudaStream_t st) {
  if (!p.fast_dct || !t.tw_v_f) return cudaErrorInvalidValue;
  return colk::vfwd_t<TM>(p, t, q, w, th, qn, wn, tn, st);
}

template <int TM>
cudaError_t ColumnOps<TM>::vback(const Params& p, const Tables& t, int mode, const VArgs& a, cudaStream_t st) {
  using namespace colk;
  VK k = make_vk(p, t);
  const bool f32 = a.Aqf != nullptr;
  const int ak = (!f32 || mode == VB_SOLVE) ? AK_F64 : (a.af_coef ? AK_F32_COEF : AK_F32_NODAL);
  const size_t sm = ak == AK_F32_COEF ? vsmem<TM>(p, 5) : vsmem<TM>(p, 5, true, ak == AK_F32_NODAL, false);
  const int g = vgrid<TM>(p);
  if (f32 && (a.dtb_nodal || !a.Awf || !a.Atf)) return cudaErrorInvalidValue;
  if (ak == AK_F32_NODAL && (!p.fast_dct || !t.tw_v_f)) return cudaErrorInvalidValue;
  switch (mode) {
    case VB_RHS: vback_ak<TM, VB_RHS>(ak, k, a, sm, g, st); break;
    case VB_STAGE1: vback_ak<TM, VB_STAGE1>(ak, k, a, sm, g, st); break;
    case VB_STAGE2: vback_ak<TM, VB_STAGE2>(ak, k, a, sm, g, st); break;
    default: vback_t<TM, VB_SOLVE, AK_F64>(k, a, sm, g, st); break;
  }
  return cudaGetLastError();
}

template <int TM>
cudaError_t ColumnOps<TM>::vpost(const Params& p, const Tables& t, const double2* Rq, const double2* Rt,
                                 const double2* w_new, double2* q_out, double2* t_out, bool zero_mean,
                                 cudaStream_t st, bool df) {
  using namespace colk;
  VK k = make_vk(p, t);
  const size_t sm = vsmem<TM>(p, 3);
  auto kern = df ? k_vpost<TM, cdfl> : k_vpost<TM, double2>;
  launch_after(kern, vgrid<TM>(p), NT, sm, st, k, Rq, Rt, w_new, q_out, t_out, zero_mean);
  return cudaGetLastError();
}

template <int TM>
cudaError_t ColumnOps<TM>::itend(const Params& p, const Tables& t, const double2* q, const double2* w,
                                 const double2* th, double2* Iq, double2* Iw, double2* It, cudaStream_t st) {
  using namespace colk;
  VK k = make_vk(p, t);
  const size_t sm = vsmem<TM>(p, 4);
  launch_after(k_itend<TM>, vgrid<TM>(p), NT, sm, st, k, q, w, th, Iq, Iw, It);
  return cudaGetLastError();
}

}  // namespace nhqg
