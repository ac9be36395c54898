// The SBP2 corrector's per-column kernels (nhqg/solver.py:909-950), templates on
// the modes per CTA like column_kernels.cuh; see corrector.cu.
#pragma once
#include <type_traits>

#include "column.cuh"
#include "engine.h"

namespace nhqg {
namespace colk {

using col::NT;
using col::Prec;

struct CK {
  int P, G, N, M;
  bool mixed;
  const double *wa, *wb;
  const double *V, *Vinv;
  col::Dct dct;
  const int *c2s_ptr, *c2s_col, *s2c_ptr, *s2c_col;
  const double *c2s_val, *s2c_val;
  const double *bcF, *bcV, *proj, *D1, *Lsbp;
  const double *c2sV, *tauVinv;  // fused dense 1-D maps (rows applied by many CTAs)
  double mu, kappa;
  const double *D1b, *Lb;  // D1 (3 diagonals) and the SBP Laplacian (5), [d][P]
  int ell_w;               // c2s / s2c as fixed-width rows, [q][P]
  const int *c2s_ecol, *s2c_ecol;
  const double *c2s_eval, *s2c_eval;
  int win_ov;              // reach of the 1-D solve's banded inverse; 0: one serial LU
};

inline CK make_ck(const Params& p, const Tables& t) {
  CK k;
  k.P = p.d.P; k.G = p.d.G; k.N = p.d.Nz; k.M = p.d.M;
  k.mixed = t.wst_a != nullptr;
  k.wa = t.wst_a; k.wb = t.wst_b;
  k.V = t.V; k.Vinv = t.Vinv;
  k.dct = make_dct(p, t);
  k.c2s_ptr = t.c2s_ptr; k.c2s_col = t.c2s_col; k.c2s_val = t.c2s_val;
  k.s2c_ptr = t.s2c_ptr; k.s2c_col = t.s2c_col; k.s2c_val = t.s2c_val;
  k.bcF = t.bcF; k.bcV = t.bcV; k.proj = t.proj; k.D1 = t.D1; k.Lsbp = t.Lsbp;
  k.c2sV = t.c2sV; k.tauVinv = t.tauVinv;
  k.mu = p.eps_sq;
  k.kappa = 1.0 / p.sigma;
  k.D1b = t.D1b; k.Lb = t.Lb;
  k.ell_w = t.ell_w;
  k.c2s_ecol = t.c2s_ecol; k.s2c_ecol = t.s2c_ecol; k.c2s_eval = t.c2s_eval; k.s2c_eval = t.s2c_eval;
  k.win_ov = 0;
  return k;
}

// Galerkin -> Chebyshev stencil of w (wbasis) or theta on tiles of type C
template <int TM, typename C>
__device__ __forceinline__ void tstencil(const CK& k, bool wbasis, C* c, const C* x) {
  const bool mixed = wbasis && k.mixed;
  for (int idx = threadIdx.x; idx < k.P * TM; idx += blockDim.x) {
    const int n = idx / TM, mm = idx - n * TM;
    C v;
    if (!mixed) {
      v = (n < k.G) ? col::gneg(x[n * TM + mm]) : col::gzero<C>();
      if (n >= 2 && n - 2 < k.G) v = gadd(v, x[(n - 2) * TM + mm]);
    } else {
      v = (n < k.G) ? x[n * TM + mm] : col::gzero<C>();
      if (n >= 1 && n - 1 < k.G) v = col::gaxpy(Prec<C>::s(__ldg(k.wa + n - 1)), x[(n - 1) * TM + mm], v);
      if (n >= 2 && n - 2 < k.G) v = col::gaxpy(Prec<C>::s(__ldg(k.wb + n - 2)), x[(n - 2) * TM + mm], v);
    }
    c[idx] = v;
  }
}
// ------------------------------------------------------------ per-mode kernels
// Tiles of type C: double2 in the plain path; cdfl (double-float on the FP32
// pipe, about 48 significant bits) in the mixed-precision path, where these
// transforms carry the state itself and FP32 would be too coarse.  Fields in
// global memory stay FP64 either way.

// out[i] = sum_j Mat[i][j] x[j] for the rows i = blockIdx.x, blockIdx.x +
// gridDim.x, ... < n, one warp per row (lane partial sums over j = lane + 32 q,
// then a fixed shuffle tree): a dense 1-D map spread over the CTAs of a
// multi-CTA kernel instead of one SM's FP64 pipe.
__device__ __forceinline__ void rows_by_ctas(const double* __restrict__ Mat, const double* __restrict__ x,
                                             double* __restrict__ out, int n) {
  if (Mat == nullptr || threadIdx.x >= 32) return;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const double* row = Mat + (size_t)i * n;
    double acc = 0.0;
    for (int j = threadIdx.x; j < n; j += 32) acc = fma(row[j], x[j], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (threadIdx.x == 0) out[i] = acc;
  }
}

// Predictor w and theta to nodal CGL values and to the SBP grid; the CTAs
// also form tb_sbp = c2s V tbp (the predictor mean temperature on the SBP grid).
// In the double-float path w runs on FP32 tiles: it enters the corrector only
// through the exchange increment sub_dt g_half w (about 1e-5 of theta, so an
// FP32 w changes theta by ~1e-12 relative), the means <w^2>, <w theta> (an
// FP32-relative error there is again scaled by sub_dt) and the nodal w of the
// next explicit RHS, whose products are FP32.  theta, the state the corrector
// carries, stays double-float.
// The double-float instantiation writes w as FP32 (wcgl_f, wsbp_f; a null
// wcgl_f skips the nodal w), the FP64 one as FP64 (wcgl, wsbp).
template <int TM, typename C>
__global__ void __launch_bounds__(NT) k_corr_pre(CK k, const double2* wp, const double2* tp,
                                                 double2* wcgl, double2* wsbp, float2* wcgl_f,
                                                 float2* wsbp_f, double2* tsbp, const double* tbp,
                                                 double* tb_sbp) {
  after_previous();
  using Cl = col::Cols<TM>;
  rows_by_ctas(k.c2sV, tbp, tb_sbp, k.P);
  using CW = typename std::conditional<std::is_same<C, cdfl>::value, float2, C>::type;
  extern __shared__ double2 sm_raw[];
  const int PT = k.P * TM;
  void* dct_base = sm_raw + 2 * PT;  // after two tiles of the widest type
  const int m0 = blockIdx.x * TM;
  Cl::tprefetch(tp, k.G, m0, k.M, sizeof(double2));  // theta, read after w's transform
  {
    CW* sw = reinterpret_cast<CW*>(sm_raw);
    CW *b0 = sw, *b1 = sw + PT;
    const col::DctSharedT<CW> ds = Cl::template dct_shared<CW>(k.dct, dct_base);
    Cl::tloadp(b0, wp, k.G, m0, k.M);
    __syncthreads();
    tstencil<TM>(k, true, b1, b0);
    __syncthreads();
    Cl::tdct(b0, b1, k.dct, ds, false, k.P);
    __syncthreads();
    if constexpr (std::is_same<CW, float2>::value) {
      if (wcgl_f != nullptr) Cl::tstorep(b0, wcgl_f, k.P, m0, k.M);
    } else {
      Cl::tstorep(b0, wcgl, k.P, m0, k.M);
    }
    Cl::tcsr(b1, b0, k.c2s_ptr, k.c2s_col, k.c2s_val, k.P);
    __syncthreads();
    if constexpr (std::is_same<CW, float2>::value) Cl::tstorep(b1, wsbp_f, k.P, m0, k.M);
    else Cl::tstorep(b1, wsbp, k.P, m0, k.M);
    __syncthreads();
  }
  C* sm = reinterpret_cast<C*>(sm_raw);
  C *b0 = sm, *b1 = sm + PT;
  const col::DctSharedT<C> ds = Cl::template dct_shared<C>(k.dct, dct_base);
  Cl::tloadp(b0, tp, k.G, m0, k.M);
  __syncthreads();
  tstencil<TM>(k, false, b1, b0);
  __syncthreads();
  Cl::tdct(b0, b1, k.dct, ds, false, k.P);
  __syncthreads();
  Cl::tcsr(b1, b0, k.c2s_ptr, k.c2s_col, k.c2s_val, k.P);
  __syncthreads();
  Cl::tstorep(b1, tsbp, k.P, m0, k.M);
}

template <int TM, typename C, typename WT>
__global__ void __launch_bounds__(NT) k_corr_sub(CK k, double2* tsbp, const WT* wsbp,
                                                 const double* g_half, double sub_dt, int last,
                                                 double2* t_out,
                                                 typename std::conditional<std::is_same<WT, float2>::value,
                                                                           float2, double2>::type* tcgl,
                                                 const double* y_mean,
                                                 double* tb_out) {
  after_previous();
  using Cl = col::Cols<TM>;
  // last substep: the corrected mean temperature tb_out = P_tau V^-1 y_mean
  if (last) rows_by_ctas(k.tauVinv, y_mean, tb_out, k.P);
  using T = typename Prec<C>::T;
  extern __shared__ double2 sm_raw[];
  C* sm = reinterpret_cast<C*>(sm_raw);
  const int PT = k.P * TM;
  // b1 and b3, side by side, are free when the transform runs: its work area
  C *b0 = sm, *b2 = sm + PT, *b1 = sm + 2 * PT, *b3 = sm + 3 * PT;
  const col::DctSharedT<C> ds = Cl::template dct_shared<C>(k.dct, sm + 4 * PT, b1);
  __shared__ C delta[2 * TM];
  const int m0 = blockIdx.x * TM;
  const int P = k.P;
  Cl::tloadp(b0, tsbp, P, m0, k.M);
  Cl::tloadp(b1, wsbp, P, m0, k.M);
  __syncthreads();
  for (int i = threadIdx.x; i < PT; i += blockDim.x) {
    const int l = i / TM;
    b0[i] = (l == 0 || l == P - 1) ? col::gzero<C>()
                                   : col::gaxpy(Prec<C>::s(-sub_dt * g_half[l]), b1[i], b0[i]);
  }
  __syncthreads();
  Cl::tcsr(b2, b0, k.s2c_ptr, k.s2c_col, k.s2c_val, P);  // y = s2c theta_sbp_new
  __syncthreads();
  if (!last || tcgl != nullptr) {
    {  // delta_j = F_j . y for j = 0, 1, re/im: 4*TM dot products, one warp each pass
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      for (int d = warp; d < 4 * TM; d += blockDim.x >> 5) {
        const int mm = d % TM, j = (d / TM) & 1, im = d / (2 * TM);
        const double* F = k.bcF + j * P;
        T acc = T(0);
        for (int l = lane; l < P; l += 32)
          acc = fma(Prec<C>::s(F[l]), im ? b2[l * TM + mm].y : b2[l * TM + mm].x, acc);
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (lane == 0) { if (im) delta[j * TM + mm].y = acc; else delta[j * TM + mm].x = acc; }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < PT; i += blockDim.x) {
      const int l = i / TM, mm = i - l * TM;
      C v = col::gaxpy(Prec<C>::s(k.bcV[l]), delta[mm], b2[i]);
      b3[i] = col::gaxpy(Prec<C>::s(k.bcV[P + l]), delta[TM + mm], v);
    }
    __syncthreads();
    if (!last) {
      Cl::tcsr(b1, b3, k.c2s_ptr, k.c2s_col, k.c2s_val, P);
      __syncthreads();
      Cl::tstorep(b1, tsbp, P, m0, k.M);
    } else {
      Cl::tstorep(b3, tcgl, P, m0, k.M);
    }
  }
  if (last) {
    __syncthreads();
    Cl::tdct(b0, b2, k.dct, ds, true, k.G);  // first G Chebyshev coefficients of V^-1 y
    __syncthreads();
    Cl::tpinv_dir(b1, b0, k.G);
    __syncthreads();
    Cl::tstorep(b1, t_out, k.G, m0, k.M);
  }
}

}  // namespace colk

template <int TM>
cudaError_t CorrColumnOps<TM>::pre(const Params& p, const Tables& t, const CorrArgs& a, bool df, double* tb_sbp,
                                   cudaStream_t st) {
  colk::CK k = colk::make_ck(p, t);
  if (tb_sbp == nullptr) k.c2sV = nullptr;  // no mean-temperature side job
  const size_t sm = 2 * (size_t)p.d.P * TM * sizeof(double2) + col::Cols<TM>::dct_smem_bytes(k.dct);
  auto kern = df ? colk::k_corr_pre<TM, cdfl> : colk::k_corr_pre<TM, double2>;
  launch_after(kern, (p.d.M + TM - 1) / TM, col::NT, sm, st, k, a.wp, a.tp, a.wcgl, a.wsbp, a.wcgl_f,
                                                   reinterpret_cast<float2*>(a.wsbp), a.tsbp, a.tbp, tb_sbp);
  return cudaGetLastError();
}

template <int TM>
cudaError_t CorrColumnOps<TM>::sub(const Params& p, const Tables& t, const CorrArgs& a, bool df,
                                   const double* g_half, double sub_dt, int last, const double* y_mean,
                                   cudaStream_t st) {
  const colk::CK k = colk::make_ck(p, t);
  const size_t sm = 4 * (size_t)p.d.P * TM * sizeof(double2) + col::Cols<TM>::dct_smem_bytes(k.dct, false, false);
  const int grid = (p.d.M + TM - 1) / TM;
  if (df) {
    auto kern = colk::k_corr_sub<TM, cdfl, float2>;
      launch_after(kern, grid, col::NT, sm, st, k, a.tsbp, reinterpret_cast<const float2*>(a.wsbp), g_half, sub_dt, last,
                                    a.t_out, a.tcgl_f, y_mean, a.tb_out);
  } else {
    auto kern = colk::k_corr_sub<TM, double2, double2>;
      launch_after(kern, grid, col::NT, sm, st, k, a.tsbp, a.wsbp, g_half, sub_dt, last, a.t_out, a.tcgl, y_mean, a.tb_out);
  }
  return cudaGetLastError();
}

}  // namespace nhqg
