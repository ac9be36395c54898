// Column engine entry points, layout kernels, reductions and the deep-grid
// form of the per-shell solve (FP64).  The per-column kernels are in
// column_kernels.cuh.
#include <algorithm>
#include <type_traits>

#include "column.cuh"
#include "engine.h"

namespace nhqg {

namespace {

using col::NT;

// =========================================================== per-shell dense solve
// FP64 form, for the depths that shell_tc.cu does not take (Nz > 257).
// w = imex_inv[shell(k)] @ rhs_w for every mode; one CTA per shell, the
// shell's matrix streams once through L1 while its modes' columns sit in
// shared memory.  NC modes per pass (compile-time, so no FMA is wasted).
template <int NC>
__device__ __forceinline__ void shell_rows(const double* __restrict__ A, const double2* xs, int G,
                                           int ld_x, double2* out, const int* modes, int M) {
  for (int i = threadIdx.x; i < G; i += blockDim.x) {
    double2 acc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = czero();
    const double* row = A + (size_t)i * G;
    for (int j = 0; j < G; ++j) {
      const double v = __ldg(row + j);
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[c] = caxpy(v, xs[j * ld_x + c], acc[c]);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) out[(size_t)i * M + modes[c]] = acc[c];
  }
}

constexpr int SHELL_NC = 8;

__global__ void __launch_bounds__(NT) k_shell(const double* mats, const int* start, const int* list,
                                              const double2* rhs, double2* out, int G, int M) {
  after_previous();
  extern __shared__ double2 xs[];  // [G][SHELL_NC]
  __shared__ int modes[SHELL_NC];
  const int s = blockIdx.x;
  const int b = start[s], e = start[s + 1];
  const double* A = mats + (size_t)s * G * G;
  for (int c0 = b; c0 < e; c0 += SHELL_NC) {
    const int nc = min(SHELL_NC, e - c0);
    if (threadIdx.x < nc) modes[threadIdx.x] = list[c0 + threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.x; i < G * nc; i += blockDim.x) {
      const int j = i / nc, c = i - j * nc;
      xs[j * SHELL_NC + c] = rhs[(size_t)j * M + modes[c]];
    }
    __syncthreads();
    switch (nc) {
      case 1: shell_rows<1>(A, xs, G, SHELL_NC, out, modes, M); break;
      case 2: shell_rows<2>(A, xs, G, SHELL_NC, out, modes, M); break;
      case 3: shell_rows<3>(A, xs, G, SHELL_NC, out, modes, M); break;
      case 4: shell_rows<4>(A, xs, G, SHELL_NC, out, modes, M); break;
      case 5: shell_rows<5>(A, xs, G, SHELL_NC, out, modes, M); break;
      case 6: shell_rows<6>(A, xs, G, SHELL_NC, out, modes, M); break;
      case 7: shell_rows<7>(A, xs, G, SHELL_NC, out, modes, M); break;
      default: shell_rows<8>(A, xs, G, SHELL_NC, out, modes, M); break;
    }
    __syncthreads();
  }
}

// =========================================================== layout kernels
// Full (Nx, Nk) planes <-> compact modes of up to three fields and th_bar, one
// warp per plane row (its 16-byte values are contiguous on both sides), five
// loads in flight per lane.  Bound by the full planes' traffic.  The gather
// also flags content outside the band.
constexpr int kRowsPerCta = 8;
constexpr int kRowLoads = 5;  // 129 columns (Nx = 256) in one batch

struct RowRef {
  int f, l, row;
  __device__ __forceinline__ RowRef(const Dims& d, const Fields3& a, int i) {
    row = i % d.Nx;
    l = i / d.Nx;
    for (f = 0; f < 2 && l >= a.levels[f]; ++f) l -= a.levels[f];
  }
};

__global__ void __launch_bounds__(32 * kRowsPerCta) k_gather(Dims d, Fields3 a, int rows, int* status) {
  after_previous();
  const int lane = threadIdx.x & 31, i = blockIdx.x * kRowsPerCta + (threadIdx.x >> 5);
  if (blockIdx.x == 0 && a.tb_in != nullptr)
    for (int l = threadIdx.x; l < d.P; l += blockDim.x) a.tb_out[l] = a.tb_in[l];
  if (i >= rows) return;
  const RowRef r(d, a, i);
  const int kx = r.row <= d.Nx / 2 ? r.row : r.row - d.Nx;
  const double2* src = a.src[r.f] + ((size_t)r.l * d.Nx + r.row) * d.Nk;
  const int keep = abs(kx) <= d.K ? min(d.K + 1, d.Nk) : 0;  // stored columns of this row
  double2* dst = a.dst[r.f] + (size_t)r.l * d.M + (size_t)(kx >= 0 ? kx : kx + d.Mr) * d.Mc;
  bool outside = false;
  for (int c0 = lane; c0 < d.Nk; c0 += 32 * kRowLoads) {
    double2 v[kRowLoads];
#pragma unroll
    for (int q = 0; q < kRowLoads; ++q) v[q] = c0 + 32 * q < d.Nk ? src[c0 + 32 * q] : czero();
#pragma unroll
    for (int q = 0; q < kRowLoads; ++q) {
      const int c = c0 + 32 * q;
      if (c < keep) dst[c] = v[q];
      else if (v[q].x != 0.0 || v[q].y != 0.0) outside = true;
    }
  }
  if (outside && status) atomicOr(status, 1 << NHQG_STATUS_BIT_OOB);
}

__global__ void __launch_bounds__(32 * kRowsPerCta) k_scatter(Dims d, Fields3 a, int rows) {
  after_previous();
  const int lane = threadIdx.x & 31, i = blockIdx.x * kRowsPerCta + (threadIdx.x >> 5);
  if (blockIdx.x == 0 && a.tb_out != nullptr)
    for (int l = threadIdx.x; l < d.P; l += blockDim.x) a.tb_out[l] = a.tb_in ? a.tb_in[l] : 0.0;
  if (i >= rows) return;
  const RowRef r(d, a, i);
  const int kx = r.row <= d.Nx / 2 ? r.row : r.row - d.Nx;
  const int keep = abs(kx) <= d.K ? min(d.K + 1, d.Nk) : 0;
  const double2* src = a.src[r.f] + (size_t)r.l * d.M + (size_t)(kx >= 0 ? kx : kx + d.Mr) * d.Mc;
  double2* dst = a.dst[r.f] + ((size_t)r.l * d.Nx + r.row) * d.Nk;
  for (int c0 = lane; c0 < d.Nk; c0 += 32 * kRowLoads) {
    double2 v[kRowLoads];
#pragma unroll
    for (int q = 0; q < kRowLoads; ++q) v[q] = c0 + 32 * q < keep ? src[c0 + 32 * q] : czero();
#pragma unroll
    for (int q = 0; q < kRowLoads; ++q)
      if (c0 + 32 * q < d.Nk) dst[c0 + 32 * q] = v[q];
  }
}

// zero the k=0 mode, Hermitian-project the ky=0 column and, in the
// full-band layout of the 3/2 rule, the ky = Nx/2 column
// (nhqg/solver.py:107-146, 993-999).  One warp per compact row; th_bar rides along.
__global__ void __launch_bounds__(32 * kRowsPerCta) k_finalize(Dims d, Fields3 a, int rows) {
  after_previous();
  const int lane = threadIdx.x & 31, i = blockIdx.x * kRowsPerCta + (threadIdx.x >> 5);
  if (blockIdx.x == 0)
    for (int l = threadIdx.x; l < d.P; l += blockDim.x) a.tb_out[l] = a.tb_in[l];
  if (i >= rows) return;
  const int r = i % d.Mr;
  int l = i / d.Mr, f = 0;
  for (; f < 2 && l >= a.levels[f]; ++f) l -= a.levels[f];
  const int cnyq = d.pad ? d.Nk - 1 : -1;
  const double2* row = a.src[f] + (size_t)l * d.M + (size_t)r * d.Mc;
  const double2* mir = a.src[f] + (size_t)l * d.M + (size_t)mirror_row(r, d.Mr) * d.Mc;
  double2* dst = a.dst[f] + (size_t)l * d.M + (size_t)r * d.Mc;
  for (int c0 = lane; c0 < d.Mc; c0 += 128) {
    double2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = c0 + 32 * q < d.Mc ? row[c0 + 32 * q] : czero();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = c0 + 32 * q;
      if (c >= d.Mc) break;
      if (c == 0 || c == cnyq) {
        // the zeroed k = 0 mode is its own mirror in the ky = 0 column
        const double2 z = mir[c];
        v[q] = (c == 0 && r == 0) ? czero() : make_double2(0.5 * (v[q].x + z.x), 0.5 * (v[q].y - z.y));
      }
      dst[c] = v[q];
    }
  }
}

// Hermitian projection of the ky=0 column (and of the ky = Nx/2 column in the
// full-band layout), in place (no k=0 zeroing)
__global__ void k_hermitian(Dims d, double2* q, double2* w, double2* th) {
  after_previous();
  const int nlev[3] = {d.P, d.G, d.G};
  double2* f3[3] = {q, w, th};
  const int half = d.Mr / 2;  // rows 1..half pair with Mr-1..Mr-half
  const int ncol = d.pad ? 2 : 1;
  const int per = ncol * (half + 1);
  const int total = (d.P + 2 * d.G) * per;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    int f = 0, j = i;
    while (j >= nlev[f] * per) { j -= nlev[f] * per; ++f; }
    const int l = j / per, rc = j - l * per;
    const int ci = rc / (half + 1), r = rc - ci * (half + 1);
    double2* col = f3[f] + (size_t)l * d.M + (ci == 0 ? 0 : d.Nk - 1);  // entries at row*Mc
    if (r == 0) {
      col[0] = make_double2(col[0].x, 0.0);
    } else {
      const int rm = mirror_row(r, d.Mr);
      const double2 a = col[(size_t)r * d.Mc], b = col[(size_t)rm * d.Mc];
      const double2 h = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
      col[(size_t)r * d.Mc] = h;
      col[(size_t)rm * d.Mc] = cconj(h);
    }
  }
}

// Horizontal mean of irfft2(a) irfft2(b) per level by Parseval: every mode of
// the half plane counts twice except the ky = 0 column, which enters through
// its Hermitian projection.  In the full-band layout of the 3/2 rule the
// means are those of the zero-padded fields (nhqg/solver.py:204-245): the
// ky = Nx/2 column is an ordinary column of the padded grid (weight 2), and
// the kx Nyquist entry of the ky = 0 column sits at kx = -Nx/2 alone, so its
// Hermitian part contributes Re(a b*)/2.  Each level is split into kParSeg segments, one CTA
// each; the last CTA of a level to finish adds the segment sums in segment
// order (deterministic) and resets the level's counter for the next launch.
// C = cdfl accumulates the per-thread sums in double-float (the mixed path;
// the FP64 pipe bounds the FP64 form on GB300); CTA totals are FP64.
constexpr int kParSeg = 4;  // 4 P CTAs: one wave on 152 SMs for P <= 257
__device__ __forceinline__ double2 as_d2(double2 v) { return v; }
__device__ __forceinline__ double2 as_d2(float2 v) { return make_double2(f2d_bits(v.x), f2d_bits(v.y)); }

template <typename C, typename TA>
__global__ void __launch_bounds__(NT) k_parseval(Dims d, const TA* a, const double2* b,
                                                 double* out, double scale, double* partials,
                                                 unsigned* counters) {
  after_previous();
  using T = typename col::Prec<C>::T;
  __shared__ double scratch[32];
  __shared__ bool is_last;
  const int l = blockIdx.y, seg = blockIdx.x;
  const TA* al = a + (size_t)l * d.M;
  const double2* bl = b + (size_t)l * d.M;
  const int chunk = (d.M + kParSeg - 1) / kParSeg;
  const int m0 = seg * chunk, m1 = min(d.M, m0 + chunk);
  // two FMAs per element on two accumulators; the half-plane weight 2 is
  // applied once
  T accr = T(0), acci = T(0);
#pragma unroll 8
  for (int m = m0 + threadIdx.x; m < m1; m += blockDim.x) {
    const C x = col::Prec<C>::in(al[m]), y = col::Prec<C>::in(bl[m]);
    accr = fma(x.x, y.x, accr);
    acci = fma(x.y, y.y, acci);
  }
  double acc;
  if constexpr (std::is_same<C, double2>::value) acc = 2.0 * (accr + acci);
  else acc = 2.0 * df_to_double(accr + acci);
  // the ky = 0 column: replace the doubled term by the Hermitian projection
  for (int r = threadIdx.x; r < d.Mr; r += blockDim.x) {
    const int m = r * d.Mc;
    if (m < m0 || m >= m1) continue;
    const int rm = mirror_row(r, d.Mr);
    const double2 x = as_d2(al[m]), xm = as_d2(al[rm * d.Mc]);
    const double2 y = bl[m], ym = bl[rm * d.Mc];
    const double xy = fma(x.x, y.x, x.y * y.y);
    if (rm == r && r != 0) {  // padded kx Nyquist (full-band layout only)
      acc += 0.5 * xy - 2.0 * xy;
      continue;
    }
    const double hx_re = 0.5 * (x.x + xm.x), hx_im = 0.5 * (x.y - xm.y);
    const double hy_re = 0.5 * (y.x + ym.x), hy_im = 0.5 * (y.y - ym.y);
    acc += fma(hx_re, hy_re, hx_im * hy_im) - 2.0 * xy;
  }
  const double tot = block_sum(acc, scratch);
  if (threadIdx.x == 0) {
    partials[(size_t)l * kParSeg + seg] = tot;
    __threadfence();
    is_last = atomicAdd(&counters[l], 1u) == kParSeg - 1;
  }
  __syncthreads();
  if (is_last && threadIdx.x == 0) {
    __threadfence();
    double sum = 0.0;
    for (int q = 0; q < kParSeg; ++q) sum += __ldcg(partials + (size_t)l * kParSeg + q);
    out[l] = sum * scale;
    counters[l] = 0u;
  }
}

// Two horizontal means in one pass over a: out_ab[l] = <a b>, out_ac[l] =
// <a c> (the corrector's <w^2> and <w theta>), same weights, order and
// arithmetic as k_parseval; partials hold two sums per (level, segment).
template <typename C, typename TA>
__global__ void __launch_bounds__(NT) k_parseval2(Dims d, const TA* a, const TA* b,
                                                  const double2* c, double* out_ab, double* out_ac,
                                                  double scale, double* partials, unsigned* counters) {
  after_previous();
  using T = typename col::Prec<C>::T;
  __shared__ double scratch[32];
  __shared__ bool is_last;
  const int l = blockIdx.y, seg = blockIdx.x;
  const TA* al = a + (size_t)l * d.M;
  const TA* bl = b + (size_t)l * d.M;
  const double2* cl = c + (size_t)l * d.M;
  const int chunk = (d.M + kParSeg - 1) / kParSeg;
  const int m0 = seg * chunk, m1 = min(d.M, m0 + chunk);
  T br = T(0), bi = T(0), cr = T(0), ci = T(0);
#pragma unroll 8
  for (int m = m0 + threadIdx.x; m < m1; m += blockDim.x) {
    const C x = col::Prec<C>::in(al[m]), y = col::Prec<C>::in(bl[m]), z = col::Prec<C>::in(cl[m]);
    br = fma(x.x, y.x, br);
    bi = fma(x.y, y.y, bi);
    cr = fma(x.x, z.x, cr);
    ci = fma(x.y, z.y, ci);
  }
  double ab, ac;
  if constexpr (std::is_same<C, double2>::value) {
    ab = 2.0 * (br + bi);
    ac = 2.0 * (cr + ci);
  } else {
    ab = 2.0 * df_to_double(br + bi);
    ac = 2.0 * df_to_double(cr + ci);
  }
  for (int r = threadIdx.x; r < d.Mr; r += blockDim.x) {
    const int m = r * d.Mc;
    if (m < m0 || m >= m1) continue;
    const int rm = mirror_row(r, d.Mr);
    const double2 x = as_d2(al[m]), xm = as_d2(al[rm * d.Mc]);
    const double2 y = as_d2(bl[m]), ym = as_d2(bl[rm * d.Mc]);
    const double2 z = cl[m], zm = cl[rm * d.Mc];
    const double xy = fma(x.x, y.x, x.y * y.y), xz = fma(x.x, z.x, x.y * z.y);
    if (rm == r && r != 0) {
      ab += 0.5 * xy - 2.0 * xy;
      ac += 0.5 * xz - 2.0 * xz;
      continue;
    }
    const double hx_re = 0.5 * (x.x + xm.x), hx_im = 0.5 * (x.y - xm.y);
    const double hy_re = 0.5 * (y.x + ym.x), hy_im = 0.5 * (y.y - ym.y);
    const double hz_re = 0.5 * (z.x + zm.x), hz_im = 0.5 * (z.y - zm.y);
    ab += fma(hx_re, hy_re, hx_im * hy_im) - 2.0 * xy;
    ac += fma(hx_re, hz_re, hx_im * hz_im) - 2.0 * xz;
  }
  const double tab = block_sum(ab, scratch);
  __syncthreads();
  const double tac = block_sum(ac, scratch);
  if (threadIdx.x == 0) {
    partials[((size_t)l * kParSeg + seg) * 2] = tab;
    partials[((size_t)l * kParSeg + seg) * 2 + 1] = tac;
    __threadfence();
    is_last = atomicAdd(&counters[l], 1u) == kParSeg - 1;
  }
  __syncthreads();
  if (is_last && threadIdx.x == 0) {
    __threadfence();
    double s1 = 0.0, s2 = 0.0;
    for (int q = 0; q < kParSeg; ++q) {
      s1 += __ldcg(partials + ((size_t)l * kParSeg + q) * 2);
      s2 += __ldcg(partials + ((size_t)l * kParSeg + q) * 2 + 1);
    }
    out_ab[l] = s1 * scale;
    out_ac[l] = s2 * scale;
    counters[l] = 0u;
  }
}

__global__ void k_zero_mode0(double2* f, int levels, int M) {
  after_previous();
  for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < levels; l += gridDim.x * blockDim.x)
    f[(size_t)l * M] = czero();
}

}  // namespace

// Modes per CTA of the column kernels.  A CTA of 256 threads wants about as many
// (level, mode) values, or most of its threads idle through the barriers of
// short columns; deep columns want several CTAs per SM (257 levels: 2 modes keep
// five FP64 tiles at 41 KB, 4 modes measured 3% and 8 modes 30% slower); and the
// grid should still give every SM work.  Measured with 2 / 4 / 8 modes: plain
// step 256^2 x 32 4.62 / 3.58 / 3.36 ms, 64^2 x 32 0.83 / 0.82 / 0.88; five mixed
// steps 96^2 x 48 3.35 / 3.06 / 3.15; explicit RHS 192^2 x 96 1.57 / 1.36 / 1.48;
// implicit solve 256^2 x 128 0.731 / 0.731 / 0.905.
int column_modes(int P, int M) {
  if (P <= 66 && M >= 8 * 4 * 152) return 8;
  if (P <= 112 && M >= 4 * 152) return 4;
  return 2;
}

cudaError_t launch_vfwd(const Params& p, const Tables& t, const double2* q, const double2* w,
                        const double2* th, double2* qn, double2* wn, double2* tn, cudaStream_t st) {
  return NHQG_BY_TM(p, ColumnOps, vfwd(p, t, q, w, th, qn, wn, tn, st));
}

cudaError_t launch_vfwd_f32(const Params& p, const Tables& t, const double2* q, const double2* w,
                            const double2* th, float2* qn, float2* wn, float2* tn, cudaStream_t st) {
  return NHQG_BY_TM(p, ColumnOps, vfwd_f32(p, t, q, w, th, qn, wn, tn, st));
}

cudaError_t launch_vback(const Params& p, const Tables& t, int mode, const VArgs& a, cudaStream_t st) {
  return NHQG_BY_TM(p, ColumnOps, vback(p, t, mode, a, st));
}

cudaError_t launch_vpost(const Params& p, const Tables& t, const double2* Rq, const double2* Rt,
                         const double2* w_new, double2* q_out, double2* t_out, bool zero_mean,
                         cudaStream_t st, bool df) {
  return NHQG_BY_TM(p, ColumnOps, vpost(p, t, Rq, Rt, w_new, q_out, t_out, zero_mean, st, df));
}

cudaError_t launch_itend(const Params& p, const Tables& t, const double2* q, const double2* w,
                         const double2* th, double2* Iq, double2* Iw, double2* It, cudaStream_t st) {
  return NHQG_BY_TM(p, ColumnOps, itend(p, t, q, w, th, Iq, Iw, It, st));
}

namespace {

__device__ __forceinline__ double2 operator*(double a, double2 b) { return make_double2(a * b.x, a * b.y); }
__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// out = base + dt * (sum_k c_k x_k), the sum taken left to right (the stage
// combinations of nhqg/solver.py:1066-1119)
template <typename T>
__global__ void k_lincomb(LinCombT<T> a) {
  after_previous();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.count; i += stride) {
    T s = a.c[0] * a.x[0][i];
    for (int k = 1; k < a.n; ++k) s = s + a.c[k] * a.x[k][i];
    a.out[i] = a.base[i] + a.dt * s;
  }
}

// K -= rate * Y per compact mode (nhqg/solver.py:1002-1009)
__global__ void k_sub_diss(double2* __restrict__ K, const double2* __restrict__ Y,
                           const double* __restrict__ rate, int levels, int M) {
  after_previous();
  const size_t n = (size_t)levels * M;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double r = rate[i % M];
    K[i] = make_double2(K[i].x - r * Y[i].x, K[i].y - r * Y[i].y);
  }
}

}  // namespace

template <typename T>
cudaError_t launch_lincomb(const LinCombT<T>& a, cudaStream_t st) {
  if (a.n < 1 || a.n > kLinCombMax) return cudaErrorInvalidValue;
  if (a.count == 0) return cudaSuccess;
  const int blocks = (int)std::min<size_t>((a.count + 255) / 256, 152 * 8);
  launch_after(k_lincomb<T>, blocks, 256, 0, st, a);
  return cudaGetLastError();
}
template cudaError_t launch_lincomb<double>(const LinCombT<double>&, cudaStream_t);
template cudaError_t launch_lincomb<double2>(const LinCombT<double2>&, cudaStream_t);

cudaError_t launch_sub_diss(const Params& p, double2* K, const double2* Y, const double* rate,
                            int levels, cudaStream_t st) {
  const size_t n = (size_t)levels * p.d.M;
  const int blocks = (int)std::min<size_t>((n + 255) / 256, 152 * 8);
  launch_after(k_sub_diss, blocks, 256, 0, st, K, Y, rate, levels, p.d.M);
  return cudaGetLastError();
}

cudaError_t launch_shell(const Params& p, const Tables& t, const Work& w, const double2* rhs_w,
                         double2* w_out, cudaStream_t st) {
  if (t.shell_fx) return launch_shell_tc(p, t, w, rhs_w, w_out, st);
  const size_t sm = (size_t)p.d.G * SHELL_NC * sizeof(double2);
  launch_after(k_shell, t.n_shells, NT, sm, st, t.shell_inv, t.shell_start, t.shell_modes, rhs_w, w_out,
                                      p.d.G, p.d.M);
  return cudaGetLastError();
}

cudaError_t launch_gather(const Params& p, const Fields3& a, int* status, cudaStream_t st) {
  const int rows = (a.levels[0] + a.levels[1] + a.levels[2]) * p.d.Nx;
  return launch_after(k_gather, (rows + kRowsPerCta - 1) / kRowsPerCta, 32 * kRowsPerCta, 0, st, p.d, a, rows,
                      status);
}

cudaError_t launch_scatter(const Params& p, const Fields3& a, cudaStream_t st) {
  const int rows = (a.levels[0] + a.levels[1] + a.levels[2]) * p.d.Nx;
  return launch_after(k_scatter, (rows + kRowsPerCta - 1) / kRowsPerCta, 32 * kRowsPerCta, 0, st, p.d, a, rows);
}

cudaError_t launch_finalize(const Params& p, const Fields3& a, cudaStream_t st) {
  const int rows = (a.levels[0] + a.levels[1] + a.levels[2]) * p.d.Mr;
  return launch_after(k_finalize, (rows + kRowsPerCta - 1) / kRowsPerCta, 32 * kRowsPerCta, 0, st, p.d, a, rows);
}

cudaError_t launch_hermitian(const Params& p, double2* q, double2* w, double2* th, cudaStream_t st) {
  launch_after(k_hermitian, 4 * 152, 256, 0, st, p.d, q, w, th);
  return cudaGetLastError();
}

cudaError_t launch_zero_mode0(const Params& p, double2* f, int levels, cudaStream_t st) {
  launch_after(k_zero_mode0, 1, 256, 0, st, f, levels, p.d.M);
  return cudaGetLastError();
}

size_t parseval_partials(int levels) { return 2 * (size_t)levels * kParSeg; }

template <typename TA>
cudaError_t parseval2_t(const Params& p, const TA* a, const TA* b, const double2* c,
                        int levels, double* out_ab, double* out_ac, Work& w, cudaStream_t st,
                        bool df) {
  const double n2 = (double)p.d.Nx * (double)p.d.Nx;
  auto kern = df ? k_parseval2<cdfl, TA> : k_parseval2<double2, TA>;
  launch_after(kern, dim3(kParSeg, levels), NT, 0, st, p.d, a, b, c, out_ab, out_ac, 1.0 / (n2 * n2), w.partials,
                                             w.counters);
  return cudaGetLastError();
}

template <typename TA>
cudaError_t parseval_t(const Params& p, const TA* a, const double2* b, int levels,
                       double* out, Work& w, cudaStream_t st, bool df) {
  const double n2 = (double)p.d.Nx * (double)p.d.Nx;
  auto kern = df ? k_parseval<cdfl, TA> : k_parseval<double2, TA>;
  launch_after(kern, dim3(kParSeg, levels), NT, 0, st, p.d, a, b, out, 1.0 / (n2 * n2), w.partials,
                                             w.counters);
  return cudaGetLastError();
}

cudaError_t launch_parseval(const Params& p, const double2* a, const double2* b, int levels,
                            double* out, Work& w, cudaStream_t st, bool df) {
  return parseval_t(p, a, b, levels, out, w, st, df);
}
cudaError_t launch_parseval(const Params& p, const float2* a, const double2* b, int levels,
                            double* out, Work& w, cudaStream_t st, bool df) {
  return parseval_t(p, a, b, levels, out, w, st, df);
}
cudaError_t launch_parseval2(const Params& p, const double2* a, const double2* b, const double2* c,
                             int levels, double* out_ab, double* out_ac, Work& w, cudaStream_t st,
                             bool df) {
  return parseval2_t(p, a, b, c, levels, out_ab, out_ac, w, st, df);
}
cudaError_t launch_parseval2(const Params& p, const float2* a, const float2* b, const double2* c,
                             int levels, double* out_ab, double* out_ac, Work& w, cudaStream_t st,
                             bool df) {
  return parseval2_t(p, a, b, c, levels, out_ab, out_ac, w, st, df);
}

}  // namespace nhqg
