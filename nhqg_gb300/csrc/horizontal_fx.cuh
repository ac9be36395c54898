// Dealiased horizontal products of the plain path in block fixed point
// (fx64.cuh), with register-resident FFTs.
//
// Same products and reference semantics as horizontal.cu (2/3 rule:
// nhqg/spectral.py:281-358; 3/2 rule: :18-50, :147-253 with the transforms at
// length N = 3 Nx/2).  The FP64 kernels are bound by the FP64 pipe (2 operations per clock
// and SM); here no transform uses it.
//
// One sequence of N = R L values belongs to a group of L lanes, R values each:
// lane l holds X[l + L e] in spectral and x[l + L e] in physical space, e < R.
// The inverse transform is an R-point DFT in registers (l fixed), the twiddles
// w_N^{a l}, then the L-point transforms over l, L = P Q, as P-point DFTs, the
// twiddles w_L^{b l}, and Q-point DFTs, with a transpose through a warp-private
// tile before each of the two; the forward transform is the transposed sequence.
// Pointwise products therefore need no data movement.  P and Q divide R, so that
// every lane holds whole sub-transforms.  R = 8 (12 where N has a factor 3) keeps
// a lane's values in 32 (48) registers: with N = 16 x 16 in two stages of 16, 64
// registers a lane left 8 warps per SM and 100 KB of code, and H1 / H2 / H3 took
// 0.62 / 1.47 / 0.77 ms at 256^2 x 257 levels.
//
// Exponents.  Every sequence carries one (fx64.cuh): H1 sets it from the
// 1-norm of its FP64 inputs and writes x1 as integers with the exponent of
// each (field, level, column); H2 aligns the columns of a row pair to the
// row's own 1-norm, transforms, multiplies, and bounds each product row by
// Cauchy-Schwarz, sum |u f| <= N |Zu|_2 |Zf|_2 (Parseval; one bit looser than
// the row's 1-norm, and known before the product is formed); H3 aligns the
// row pairs of a column the same way and returns to FP64.  H2 and H3 hold sequences
// of up to 2^62 in 1-norm, twice H1's, which halves their unit: with H1's range in all
// three the Jacobian at 256^2 was 5.8e-16 off against 5.5e-16 in FP64 (white planes),
// and 2.8e-16 so; every other length and form is below FP64 too, by up to 4.  Only the wavenumber
// factors run in FP64.  All reductions are integer or fixed-order, so results
// do not depend on the launch shape.
//
// Measured, one evaluation: 256^2 x 257 levels 8.8 -> 2.1 ms (H1 1.51 -> 0.43,
// H2 5.53 -> 1.07, H3 1.73 -> 0.60), 192^2 x 97 2.09 -> 0.66, 128^2 x 81 under the
// 3/2 rule 1.73 -> 0.65, full planes 256^2 x 65 2.56 -> 0.65.  H2 issues in 60% of
// the cycles (16 warps per SM, limited by registers and shared memory).
//
// Scaling: irfft2's 1/(N Nx) of both factors of a product rides on the
// velocity factor (kx_s, ky_s, host tables), the sponge's on its table.
#pragma once
#include <utility>

#include "engine.h"
#include "fx64.cuh"

namespace nhqg {
namespace hfx {

using namespace fx;

template <typename F, int... I>
__device__ __forceinline__ void sfor_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F>
__device__ __forceinline__ void sfor(F&& f) {
  sfor_impl(f, std::make_integer_sequence<int, N>{});
}

constexpr unsigned kFull = 0xffffffffu;

// In-register DFT of length R over x[O + S i], natural order in and out,
// R = P Q as y[a + Q b] = sum_p w_P^{b p} w_R^{a p} sum_q w_Q^{a q} x[p + P q].
template <int R, int SGN>
struct Dft {
  static constexpr int P = (R % 4 == 0 && R > 8) ? 4 : 2;
  static constexpr int Q = R / P;
  template <int O, int S>
  __device__ __forceinline__ static void run(cfx* x) {
    sfor<P>([&](auto p) { Dft<Q, SGN>::template run<O + S * decltype(p)::value, S * P>(x); });
    sfor<P>([&](auto p) {
      sfor<Q>([&](auto a) {
        constexpr int pp = decltype(p)::value, aa = decltype(a)::value;
        x[O + S * (pp + P * aa)] = rot<R, aa * pp, SGN>(x[O + S * (pp + P * aa)]);
      });
    });
    sfor<Q>([&](auto a) { Dft<P, SGN>::template run<O + S * P * decltype(a)::value, S>(x); });
    cfx t[R];
    sfor<Q>([&](auto a) {
      sfor<P>([&](auto b) {
        constexpr int aa = decltype(a)::value, bb = decltype(b)::value;
        t[aa + Q * bb] = x[O + S * (bb + P * aa)];
      });
    });
    sfor<R>([&](auto i) { x[O + S * decltype(i)::value] = t[decltype(i)::value]; });
  }
};
template <int SGN>
struct Dft<2, SGN> {
  template <int O, int S>
  __device__ __forceinline__ static void run(cfx* x) {
    const cfx a = x[O], b = x[O + S];
    x[O] = cadd(a, b);
    x[O + S] = csub(a, b);
  }
};
template <int SGN>
struct Dft<3, SGN> {
  template <int O, int S>
  __device__ __forceinline__ static void run(cfx* x) {
    const cfx x0 = x[O], x1 = x[O + S], x2 = x[O + 2 * S];
    const cfx sp = cadd(x1, x2), df = csub(x1, x2);
    const cfx m = cfx{x0.x - ((sp.x + 1) >> 1), x0.y - ((sp.y + 1) >> 1)};
    constexpr long long h = sin48(16);  // sqrt(3)/2
    const cfx d = cfx{rmul(df.x, h), rmul(df.y, h)};
    x[O] = cadd(x0, sp);
    // m + SGN i d, m - SGN i d
    const cfx p = cfx{m.x - d.y, m.y + d.x}, q = cfx{m.x + d.y, m.y - d.x};
    x[O + S] = SGN > 0 ? p : q;
    x[O + 2 * S] = SGN > 0 ? q : p;
  }
};
template <int SGN>
struct Dft<4, SGN> {
  template <int O, int S>
  __device__ __forceinline__ static void run(cfx* x) {
    const cfx a0 = x[O], a1 = x[O + S], a2 = x[O + 2 * S], a3 = x[O + 3 * S];
    const cfx t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3);
    const cfx t3 = rot<4, 1, SGN>(csub(a1, a3));
    x[O] = cadd(t0, t2);
    x[O + 2 * S] = csub(t0, t2);
    x[O + S] = cadd(t1, t3);
    x[O + 3 * S] = csub(t1, t3);
  }
};

// Transforms of one lane group; T is its transpose tile, tw the shared twiddles
// exp(+2 pi i a l / N) at a L + l, followed by exp(+2 pi i b q / L) at b Q + q.
template <int R_, int L_, int P_, int Q_>
struct Lane {
  static constexpr int R = R_, L = L_, P = P_, Q = Q_, N = R * L;
  static_assert(P * Q == L && R % P == 0 && R % Q == 0 && L <= 32, "whole sub-transforms per lane");
  static constexpr int LS = L > 16 ? 32 : (L > 8 ? 16 : (L > 4 ? 8 : 4));  // lanes of a group
  static constexpr int G = 32 / LS;                                        // groups per warp
  static constexpr int CB = 8;                                             // groups per CTA
  static constexpr int W = CB / G;                                         // warps per CTA
  static constexpr int MINB = R == 8 && L == 32 ? 2 : 12 / W;              // 16 or 12 warps per SM
  static constexpr int NA = R / P, NC = R / Q;  // P- and Q-point transforms per lane
  // row strides of the two transposes, so that eight consecutive lanes (one
  // phase of a 16-byte access) fall on distinct bank groups
  static constexpr int SA = L + ((Q - L) % 8 + 8) % 8;
  static constexpr int SCm = Q == 4 ? 2 : (Q == 2 ? 4 : 3);
  static constexpr int SC = R * P + ((SCm - R * P) % 8 + 8) % 8;
  static constexpr int TILE0 = R * SA > (Q > 1 ? Q * SC : 0) ? R * SA : Q * SC;
  static constexpr int TILE = LS == 4 ? TILE0 + ((4 - TILE0) % 8 + 8) % 8 : TILE0;
  static constexpr int TW = N + P * Q;

  struct Tables {
    const int4* a;  // ch, cl, dh, dl
    const int2* b;  // nh, nl
    __device__ __forceinline__ Tw at(int i) const {
      const int4 u = a[i];
      const int2 v = b[i];
      return Tw{u.x, u.y, u.z, u.w, v.x, v.y};
    }
  };

  __device__ __forceinline__ static void inv(cfx* x, cfx* T, const Tables& tw, int l) {
    const bool on = l < L;
    const int t = on ? l : 0, l0 = t % Q, a0 = t / Q;
    Dft<R, +1>::template run<0, 1>(x);
    sfor<R>([&](auto aa) {
      constexpr int A = decltype(aa)::value;
      if constexpr (A > 0) x[A] = cmul<false>(x[A], tw.at(A * L + t));
      if (on) T[A * SA + t] = x[A];
    });
    __syncwarp();
    cfx z[R];
    sfor<NA>([&](auto kk) {
      sfor<P>([&](auto pp) {
        constexpr int k = decltype(kk)::value, q = decltype(pp)::value;
        z[k * P + q] = T[(a0 + P * k) * SA + l0 + Q * q];
      });
    });
    __syncwarp();
    sfor<NA>([&](auto kk) { Dft<P, +1>::template run<decltype(kk)::value * P, 1>(z); });
    if constexpr (Q > 1) {
      sfor<NA>([&](auto kk) {
        sfor<P>([&](auto bb) {
          constexpr int k = decltype(kk)::value, b = decltype(bb)::value;
          if constexpr (b > 0) z[k * P + b] = cmul<false>(z[k * P + b], tw.at(N + b * Q + l0));
          if (on) T[l0 * SC + a0 + P * k + R * b] = z[k * P + b];
        });
      });
      __syncwarp();
      sfor<NC>([&](auto mm) {
        sfor<Q>([&](auto qq) {
          constexpr int m = decltype(mm)::value, q = decltype(qq)::value;
          z[m * Q + q] = T[q * SC + t + L * m];
        });
      });
      __syncwarp();
      sfor<NC>([&](auto mm) { Dft<Q, +1>::template run<decltype(mm)::value * Q, 1>(z); });
      sfor<NC>([&](auto mm) {
        sfor<Q>([&](auto bb) {
          constexpr int m = decltype(mm)::value, b = decltype(bb)::value;
          x[m + NC * b] = z[m * Q + b];
        });
      });
    } else {
      sfor<NA>([&](auto kk) {
        sfor<P>([&](auto bb) {
          constexpr int k = decltype(kk)::value, b = decltype(bb)::value;
          x[k + NA * b] = z[k * P + b];
        });
      });
    }
  }

  __device__ __forceinline__ static void fwd(cfx* x, cfx* T, const Tables& tw, int l) {
    const bool on = l < L;
    const int t = on ? l : 0, l0 = t % Q, a0 = t / Q;
    cfx z[R];
    if constexpr (Q > 1) {
      sfor<NC>([&](auto mm) {
        sfor<Q>([&](auto bb) {
          constexpr int m = decltype(mm)::value, b = decltype(bb)::value;
          z[m * Q + b] = x[m + NC * b];
        });
      });
      sfor<NC>([&](auto mm) { Dft<Q, -1>::template run<decltype(mm)::value * Q, 1>(z); });
      if (on) {
        sfor<NC>([&](auto mm) {
          sfor<Q>([&](auto qq) {
            constexpr int m = decltype(mm)::value, q = decltype(qq)::value;
            T[q * SC + t + L * m] = z[m * Q + q];
          });
        });
      }
      __syncwarp();
      sfor<NA>([&](auto kk) {
        sfor<P>([&](auto bb) {
          constexpr int k = decltype(kk)::value, b = decltype(bb)::value;
          z[k * P + b] = T[l0 * SC + a0 + P * k + R * b];
          if constexpr (b > 0) z[k * P + b] = cmul<true>(z[k * P + b], tw.at(N + b * Q + l0));
        });
      });
      __syncwarp();
    } else {
      sfor<NA>([&](auto kk) {
        sfor<P>([&](auto bb) {
          constexpr int k = decltype(kk)::value, b = decltype(bb)::value;
          z[k * P + b] = x[k + NA * b];
        });
      });
    }
    sfor<NA>([&](auto kk) { Dft<P, -1>::template run<decltype(kk)::value * P, 1>(z); });
    if (on) {
      sfor<NA>([&](auto kk) {
        sfor<P>([&](auto pp) {
          constexpr int k = decltype(kk)::value, q = decltype(pp)::value;
          T[(a0 + P * k) * SA + l0 + Q * q] = z[k * P + q];
        });
      });
    }
    __syncwarp();
    sfor<R>([&](auto aa) {
      constexpr int A = decltype(aa)::value;
      x[A] = T[A * SA + t];
      if constexpr (A > 0) x[A] = cmul<true>(x[A], tw.at(A * L + t));
    });
    __syncwarp();
    Dft<R, -1>::template run<0, 1>(x);
  }
};

// max / sum over the LS lanes of a group
template <int LS>
__device__ __forceinline__ int gmax(int v) {
  for (int o = LS / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
template <int LS>
__device__ __forceinline__ unsigned gsum(unsigned v) {
  for (int o = LS / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
template <int LS>
__device__ __forceinline__ float gsumf(float v) {  // the same order in every lane pair: deterministic
  for (int o = LS / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Align NE values per lane, z[i] held at exponent e[i] (|re|, |im| <= 2^62), to one
// exponent E with |re| + |im| summed over the group's sequence below 2^(E + 1): the
// transforms take sequences up to 2^62 (fx64.cuh), of which H1, whose inputs come from
// FP64 in 61 bits, uses half.  E is not taken below the largest e: the inputs hold no
// finer units.
template <int LS, int NE>
__device__ __forceinline__ int align(cfx* z, const int* e) {
  int em = kEZero;
  sfor<NE>([&](auto i) { em = max(em, e[decltype(i)::value]); });
  em = gmax<LS>(em);
  if (em >= kENanTest) return kENan;
  unsigned s = 0;
  sfor<NE>([&](auto ii) {
    constexpr int i = decltype(ii)::value;
    s += cterm(z[i], min(31, em - e[i]));
  });
  s = gsum<LS>(s);
  const int E = max(em, em - (kBits - 40) + bitlen(s) - 1);
  sfor<NE>([&](auto ii) {
    constexpr int i = decltype(ii)::value;
    const int d = min(62, E - e[i]);
    z[i].x = shr_round(z[i].x, d);
    z[i].y = shr_round(z[i].y, d);
  });
  return E;
}
// sum over the sequence of an upper bound of |re|^2 + |im|^2 in units 2^64
template <int LS, int NE>
__device__ __forceinline__ float norm2(const cfx* z) {
  float s = 0.f;
  sfor<NE>([&](auto ii) {
    constexpr int i = decltype(ii)::value;
    const float a = (float)(abs((int)(z[i].x >> 32)) + 1), b = (float)(abs((int)(z[i].y >> 32)) + 1);
    s = fmaf(a, a, fmaf(b, b, s));
  });
  return gsumf<LS>(s);
}

struct HX {
  int Nx, Nk, K, Mr, Mc, M, levels;
  int rows_in, cols_in;
  bool full_in, full_out;
  int form, nf1, ng;
  int stage;  // raw fields that H1 stages at a time
  bool sponge, eta, psi_derived;
  const double2 *psi, *q, *w, *th;
  const double *kx, *ky;      // [Nx], [Nk]
  const double *kx_s, *ky_s;  // the same times 1/(N Nx)^2
  const double* inv_denom;    // compact [M]
  const double2* eta_c;       // compact [M]
  const long long *sponge_fx, *eta_fx;  // [N*N] at exponents sponge_e, eta_e[row pair]
  int sponge_e;
  const int* eta_e;
  const int* tw;              // 6 ints per exp(+2 pi i k / N), k < N
  cfx *x1, *x2;
  int *e1, *e2;
  double2 *Aq, *Aw, *Ath;
};

// H1 -> H2 [f][lev][x/2][c][x%2], exponents [f][lev][c];
// H2 -> H3 [g][lev][x/2][c][x%2], exponents [g][lev][x/2]
template <int N>
__device__ __forceinline__ size_t pidx(const HX& k, int f, int lev, int pair, int c, int cols) {
  return ((((size_t)f * k.levels + lev) * (N / 2) + pair) * cols + c) * 2;
}

template <typename F>
__device__ __forceinline__ typename F::Tables load_twiddles(const HX& k, int4* ta, int2* tb) {
  for (int i = threadIdx.x; i < F::TW; i += blockDim.x) {
    const int b = i - F::N;
    const int e = b < 0 ? (i / F::L) * (i % F::L) : F::R * (b / F::Q) * (b % F::Q);
    const int* t = k.tw + 6 * (e % F::N);
    ta[i] = make_int4(t[0], t[1], t[2], t[3]);
    tb[i] = make_int2(t[4], t[5]);
  }
  return typename F::Tables{ta, tb};
}
// the tables and the groups' transpose tiles lead the dynamic shared memory
template <typename F>
__host__ __device__ constexpr size_t table_bytes() {
  return (size_t)F::TW * sizeof(int4) + ((size_t)F::TW * sizeof(int2) + 15) / 16 * 16;
}
template <typename F>
__host__ __device__ constexpr size_t head_bytes() { return table_bytes<F>() + (size_t)F::CB * F::TILE * sizeof(cfx); }
template <typename F>
struct Head {
  int4* ta;
  int2* tb;
  cfx* T;
  cfx* rest;
  __device__ __forceinline__ explicit Head(unsigned char* sm) {
    ta = reinterpret_cast<int4*>(sm);
    tb = reinterpret_cast<int2*>(ta + F::TW);
    T = reinterpret_cast<cfx*>(sm + table_bytes<F>());
    rest = T + F::CB * F::TILE;
  }
};

// full-layout row of transform position kpos (-1 in the padding), and the
// input row of a full-layout row (compact or full planes; -1: not stored)
template <int N>
__device__ __forceinline__ int pos_row(const HX& k, int kpos) {
  if (kpos < k.Nx / 2) return kpos;
  if (kpos >= N - k.Nx / 2) return kpos - (N - k.Nx);
  return -1;
}
__device__ __forceinline__ int kept_row(const HX& k, int kf) {
  if (kf < 0) return -1;
  if (kf <= k.K) return kf;
  if (kf >= k.Nx - (k.Mr - k.K - 1)) return kf - (k.Nx - k.Mr);
  return -1;
}

// ---------------------------------------------------------------- H1
// CB columns per CTA, one lane group each, and two raw fields of (psi, q, w,
// theta), staged through shared memory; one where two would leave one CTA per SM
// (full 256^2 planes, 65 levels: 0.25 ms with two, 0.19 with one; the compact
// rectangle, 257 levels: 0.44 with two, 0.52 with one) or the grid is small.
template <typename F>
__global__ void __launch_bounds__(32 * F::W, F::L == 32 ? 2 : 1) k_h1x(HX k) {
  constexpr int N = F::N, R = F::R, L = F::L, LS = F::LS, G = F::G, CB = F::CB, TS = CB + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Head<F> hd(smem_raw);
  double2* tile = reinterpret_cast<double2*>(hd.rest);  // [stage][rows_in][TS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / LS, l = lane % LS;
  const int lev = blockIdx.y, c0 = blockIdx.x * CB, ncb = min(CB, k.cols_in - c0);
  const auto tw = load_twiddles<F>(k, hd.ta, hd.tb);
  const int cc = warp * G + g, c = c0 + cc;
  const bool live = cc < ncb;
  cfx* Tg = hd.T + (size_t)cc * F::TILE;
  after_previous();
  const size_t plane = (size_t)k.rows_in * k.cols_in;
  const double ky = live ? k.ky[c] : 0.0, kys = live ? k.ky_s[c] : 0.0;
  const size_t lev0 = (size_t)lev * plane;
  const int raw0 = blockIdx.z * k.stage;
  auto value = [&](int raw, int r, int c2) {
    const size_t off = lev0 + (size_t)r * k.cols_in + c2;
    if (raw == 0) return k.psi_derived ? cscale(k.q[off], -k.inv_denom[r * k.Mc + c2]) : k.psi[off];
    if (raw > 1) return raw == 2 ? k.w[off] : k.th[off];
    double2 v = k.q[off];
    if (k.eta) {
      const double2 e = k.eta_c[r * k.Mc + c2];
      v = make_double2(v.x + e.x, v.y + e.y);
    }
    return v;
  };
  for (int i = threadIdx.x; i < k.rows_in * CB; i += blockDim.x) {
    const int r = i / CB, cc2 = i % CB, c2 = c0 + cc2;
    double2 v0 = czero(), v1 = czero();
    if (cc2 < ncb) {
      v0 = value(raw0, r, c2);
      if (k.stage == 2) v1 = value(raw0 + 1, r, c2);
    }
    tile[(size_t)r * TS + cc2] = v0;
    if (k.stage == 2) tile[((size_t)k.rows_in + r) * TS + cc2] = v1;
  }
  __syncthreads();
  // output fields of these raw fields: flux u, v | q | w | theta, Jacobian f_x, f_y each
  const int rl = raw0 + k.stage - 1;
  const int f0 = k.form == HF_FLUX ? (raw0 == 0 ? 0 : raw0 + 1) : 2 * raw0;
  const int f1 = k.form == HF_FLUX ? rl + 2 : 2 * rl + 2;
#pragma unroll 1
  for (int f = f0; f < f1; ++f) {
    const int raw = k.form == HF_FLUX ? (f < 2 ? 0 : f - 1) : f >> 1;
    int der = 0;  // 0 none, 1 i kx, 2 i ky, 3 -i ky; velocity factors scaled
    if (k.form == HF_FLUX) der = f == 0 ? 3 : (f == 1 ? 1 : 0);
    else der = (f & 1) ? 2 : 1;
    const bool vel = raw == 0 && der != 0;  // velocity factor: carries the scale
    const double2* t = tile + (size_t)(raw - raw0) * k.rows_in * TS + cc;
    const double* kxt = vel ? k.kx_s : k.kx;
    const double kyf = (der == 3 ? -1.0 : 1.0) * (vel ? kys : ky);
    double2 v[R];
    int em = 1;
    sfor<R>([&](auto jj) {
      constexpr int j = decltype(jj)::value;
      const int kf = (live && l < L) ? pos_row<N>(k, l + L * j) : -1;
      const int r = k.full_in ? kf : kept_row(k, kf);
      v[j] = czero();
      if (r >= 0) {
        const double2 a = t[(size_t)r * TS];
        if (der == 0) {
          v[j] = a;
        } else {
          const double s = der == 1 ? kxt[kf] : kyf;
          v[j] = make_double2(-s * a.y, s * a.x);
        }
      }
      em = max(em, max(dexp(v[j].x), dexp(v[j].y)));
    });
    em = gmax<LS>(em);
    // columns of zeros (planes beyond the 2/3 band) need no transform: their
    // exponent tells H2 so (1 is the exponent of the subnormals too)
    if (__all_sync(kFull, em == 1)) {
      unsigned long long any = 0;
      sfor<R>([&](auto jj) { any |= dbits(v[decltype(jj)::value].x) | dbits(v[decltype(jj)::value].y); });
      if (!__any_sync(kFull, (any << 1) != 0)) {
        if (live && l == 0) k.e1[((size_t)f * k.levels + lev) * k.cols_in + c] = kEZero;
        continue;
      }
    }
    unsigned s = 0;
    sfor<R>([&](auto jj) {
      constexpr int j = decltype(jj)::value;
      s += dterm(v[j].x, em) + dterm(v[j].y, em);
    });
    s = gsum<LS>(s);
    int E = dbound(em, s);
    cfx x[R];
    sfor<R>([&](auto jj) {
      constexpr int j = decltype(jj)::value;
      x[j] = cfx{to_fx(v[j].x, E), to_fx(v[j].y, E)};
    });
    if (em == 0x7ff) E = kENan;
    F::inv(x, Tg, tw, l);
    if (live && l < L) {
      sfor<R>([&](auto bb) {
        constexpr int b = decltype(bb)::value;
        const int xx = l + L * b;
        k.x1[pidx<N>(k, f, lev, xx >> 1, c, k.cols_in) + (xx & 1)] = x[b];
      });
      if (l == 0) k.e1[((size_t)f * k.levels + lev) * k.cols_in + c] = E;
    }
  }
}

// ---------------------------------------------------------------- H2
// One lane group per row pair (a, b), Z = Xa + i Xb.  The two velocity factors
// stay in the group's own shared memory in physical space.
template <typename F, int FORM, bool SP>
__global__ void __launch_bounds__(32 * F::W, F::MINB) k_h2x(HX k) {
  constexpr int N = F::N, R = F::R, L = F::L, LS = F::LS, G = F::G, CB = F::CB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Head<F> hd(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / LS, l = lane % LS, gi = warp * G + g;
  const int lev = blockIdx.y;
  const int pp = blockIdx.x * CB + gi;
  const bool live = pp < N / 2;
  const int pair = live ? pp : 0;
  cfx* Tg = hd.T + (size_t)gi * F::TILE;
  cfx* Us = hd.rest + (size_t)gi * 2 * R * LS + l;  // element e at e LS
  cfx* Vs = Us + R * LS;
  const auto tw = load_twiddles<F>(k, hd.ta, hd.tb);
  __syncthreads();
  after_previous();
  const int cols = k.cols_in;

  auto prefetch = [&](int f) {
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(k.x1 + pidx<N>(k, f, lev, pair, 0, cols));
    const uintptr_t end = a0 + (uintptr_t)cols * 2 * sizeof(cfx);
    for (uintptr_t a = (a0 & ~uintptr_t(127)) + 128 * (uintptr_t)l; a < end; a += 128 * LS)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
  };
  // physical values of field f's row pair, their exponent and 2-norm bound
  auto load = [&](int f, cfx* x, int& E, float& nrm) {
    const cfx* base = k.x1 + pidx<N>(k, f, lev, pair, 0, cols);
    const int* eb = k.e1 + ((size_t)f * k.levels + lev) * cols;
    int e[R];
    sfor<R>([&](auto jj) {
      constexpr int j = decltype(jj)::value;
      const int c = l + L * j;
      const bool mir = c > N - cols;  // Hermitian extension
      const int m = mir ? N - c : c;
      x[j] = cfx{0, 0};
      e[j] = kEZero;
      if (l < L && m < cols) {
        const cfx A = base[2 * m], B = base[2 * m + 1];
        e[j] = eb[m];
        if (e[j] == kEZero) return;  // not written by H1
        if (c < cols) x[j] = (c == 0 || c == N / 2) ? cfx{A.x, B.x} : cfx{A.x - B.y, A.y + B.x};
        else x[j] = cfx{A.x + B.y, B.x - A.y};
      }
    });
    E = align<LS, R>(x, e);
    nrm = sqrtf(norm2<LS, R>(x)) * 1.001f;  // units 2^32
    F::inv(x, Tg, tw, l);
  };
  // exponent E of a product row of factors (Ea, na) and (Eb, nb), whose 1-norm is below
  // N na nb 2^64 2^(Ea + Eb - 2 kBits) and, as in align, may reach 2^(E + 1)
  auto pexp = [&](int Ea, float na, int Eb, float nb) {
    const int E = Ea + Eb + fexp((float)N * na * nb) + 64 - 2 * kBits - 1;
    return (Ea >= kENanTest || Eb >= kENanTest) ? kENan : max(E, Ea + Eb + kMinShift - kBits);
  };
  // spectra of the two rows at the kept columns of output gout
  auto split_store = [&](const cfx* x, int gout, int E) {
    const int src = g * LS + (l < L ? (L - l) % L : 0);
    cfx* out = k.x2 + pidx<N>(k, gout, lev, pair, 0, k.Mc);
    sfor<R / 2 + 1>([&](auto jj) {
      constexpr int j = decltype(jj)::value;
      if (L * j < k.Mc) {
        constexpr int jm = R - 1 - j, j0 = (R - j) % R;
        cfx B;
        B.x = __shfl_sync(kFull, x[jm].x, src);
        B.y = __shfl_sync(kFull, x[jm].y, src);
        if (l == 0) B = x[j0];
        const cfx A = x[j];
        const int c = l + L * j;
        if (live && l < L && c < k.Mc) {
          out[2 * c] = cfx{(A.x + B.x + 1) >> 1, (A.y - B.y + 1) >> 1};
          out[2 * c + 1] = cfx{(A.y + B.y + 1) >> 1, (B.x - A.x + 1) >> 1};
        }
      }
    });
    if (live && l == 0) k.e2[((size_t)gout * k.levels + lev) * (N / 2) + pair] = E;
  };

  // One copy of each transform's code: fields run through one loop (0, 1 the
  // velocity factors), so that the unrolled transforms fit the instruction cache.
  cfx x[R], y[R];
  int Eu = 0, Ev = 0, Ey = 0;
  float nu = 0.f, nv = 0.f, ny = 0.f;
  // after the velocity factors, this CTA's share of the other input fields
  const int per = (k.nf1 - 2) / gridDim.z, f0 = 2 + per * blockIdx.z, f1 = f0 + per;
#pragma unroll 1
  for (int f = 0; f < f1; ++f) {
    int E;
    float nrm;
    if (f == 2) f = f0;
    if (f + 1 < f1) prefetch(f == 1 ? f0 : f + 1);
    load(f, x, E, nrm);
    if (f < 2) {
      cfx* W = f ? Vs : Us;
      sfor<R>([&](auto b) { W[decltype(b)::value * LS] = x[decltype(b)::value]; });
      if (f) { Ev = E; nv = nrm; } else { Eu = E; nu = nrm; }
      continue;
    }
    int nout = 1, g0 = 0;
    if constexpr (FORM == HF_FLUX) {
      nout = SP ? 3 : 2;
      g0 = f - 2;
    } else {
      if ((f & 1) == 0) {  // f_x waits in registers for f_y
        sfor<R>([&](auto b) { y[decltype(b)::value] = x[decltype(b)::value]; });
        Ey = E;
        ny = nrm;
        continue;
      }
      g0 = (f - 3) >> 1;
    }
#pragma unroll 1
    for (int h = 0; h < nout; ++h) {
      int Ep, gout;
      if constexpr (FORM == HF_FLUX) {
        gout = h < 2 ? 2 * g0 + h : 6 + g0;
        if (!SP || h < 2) {  // F(u f), then F(v f)
          const cfx* W = h ? Vs : Us;
          const int Ew = h ? Ev : Eu;
          Ep = pexp(Ew, h ? nv : nu, E, nrm);
          const int rs = prod_shift(Ep, Ew, E);
          sfor<R>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            const cfx w = W[b * LS];
            y[b] = cfx{mul_shift(w.x, x[b].x, rs), mul_shift(w.y, x[b].y, rs)};
          });
        } else {
          // sigma (f - eta), |sigma| < 2^sponge_e: the product row's 1-norm is
          // below sqrt(2N) 2^sponge_e |f - eta|_2, the norm taken after the
          // subtraction (eta may exceed q by orders of magnitude)
          const bool sub = g0 == 0 && k.eta;
          const int ee = sub ? k.eta_e[pair] : kEZero;
          const int Es = E >= kENanTest ? kENan : (sub ? max(E, ee) + 1 : E);
          const int df = min(62, Es - E), de = min(62, Es - ee);
          const size_t p0 = (size_t)(2 * pair) * N + (l < L ? l : 0);
          sfor<R>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            y[b] = l < L ? x[b] : cfx{0, 0};
            if (sub && l < L) {
              y[b].x = shr_round(x[b].x, df) - shr_round(k.eta_fx[p0 + L * b], de);
              y[b].y = shr_round(x[b].y, df) - shr_round(k.eta_fx[p0 + N + L * b], de);
            }
          });
          const float nd = sqrtf(norm2<LS, R>(y)) * sqrtf(2.f * N) * 1.001f;
          Ep = k.sponge_e + Es + fexp(nd) + 32 - kBits - 1;
          Ep = Es >= kENanTest ? kENan : max(Ep, k.sponge_e + Es + kMinShift - kBits);
          const int rs = prod_shift(Ep, k.sponge_e, Es);
          sfor<R>([&](auto bb) {
            constexpr int b = decltype(bb)::value;
            y[b].x = mul_shift(k.sponge_fx[p0 + L * b], y[b].x, rs);
            y[b].y = mul_shift(k.sponge_fx[p0 + N + L * b], y[b].y, rs);
          });
        }
      } else {  // J_f = psi_x f_y - psi_y f_x
        gout = g0;
        const int E1 = pexp(Eu, nu, E, nrm), E2 = pexp(Ev, nv, Ey, ny);
        Ep = max(E1, E2) >= kENanTest ? kENan : max(E1, E2) + 1;
        const int r1 = prod_shift(Ep, Eu, E), r2 = prod_shift(Ep, Ev, Ey);
        sfor<R>([&](auto bb) {
          constexpr int b = decltype(bb)::value;
          const cfx px = Us[b * LS], py = Vs[b * LS];
          y[b] = cfx{mul_shift(px.x, x[b].x, r1) - mul_shift(py.x, y[b].x, r2),
                     mul_shift(px.y, x[b].y, r1) - mul_shift(py.y, y[b].y, r2)};
        });
      }
      F::fwd(y, Tg, tw, l);
      split_store(y, gout, Ep);
    }
  }
}

// ---------------------------------------------------------------- H3
template <typename F>
__global__ void __launch_bounds__(32 * F::W, F::MINB) k_h3x(HX k) {
  constexpr int N = F::N, R = F::R, L = F::L, LS = F::LS, G = F::G, CB = F::CB, TS = CB + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Head<F> hd(smem_raw);
  double2* tile = reinterpret_cast<double2*>(hd.rest);  // [Mr][TS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane / LS, l = lane % LS;
  const int lev = blockIdx.y, c0 = blockIdx.x * CB, ncb = min(CB, k.Mc - c0);
  const int cc = warp * G + g, c = c0 + cc;
  const bool live = cc < ncb;
  const int cr = live ? c : c0;  // dead groups transform a live column and discard it
  cfx* Tg = hd.T + (size_t)cc * F::TILE;
  const auto tw = load_twiddles<F>(k, hd.ta, hd.tb);
  __syncthreads();
  after_previous();
  const double ky = k.ky[cr];
  auto load = [&](int gi, cfx* x) {
    int e[R];
    const int* eb = k.e2 + ((size_t)gi * k.levels + lev) * (N / 2);
    sfor<R>([&](auto bb) {
      constexpr int b = decltype(bb)::value;
      x[b] = cfx{0, 0};
      e[b] = kEZero;
      if (l < L) {
        const int xx = l + L * b;
        x[b] = k.x2[pidx<N>(k, gi, lev, xx >> 1, cr, k.Mc) + (xx & 1)];
        e[b] = eb[xx >> 1];
      }
    });
    const int E = align<LS, R>(x, e);
    F::fwd(x, Tg, tw, l);
    return E;
  };
  const int f = blockIdx.z;  // q, w, theta
  double2 v[R];  // values at rows l + L j
  cfx x[R];
  const bool flux = k.form == HF_FLUX;
  const int npart = flux ? (k.sponge ? 3 : 2) : 1;
#pragma unroll 1
  for (int h = 0; h < npart; ++h) {
    const int gi = flux ? (h < 2 ? 2 * f + h : 6 + f) : f;
    const int E = load(gi, x);
    sfor<R>([&](auto jj) {
      constexpr int j = decltype(jj)::value;
      const int kf = l < L ? pos_row<N>(k, l + L * j) : -1;
      if (kept_row(k, kf) >= 0) {
        const double2 d = make_double2(from_fx(x[j].x, E), from_fx(x[j].y, E));
        if (!flux) {
          v[j] = d;
        } else if (h == 0) {  // i kx F(u f)
          const double kx = k.kx[kf];
          v[j] = make_double2(-kx * d.y, kx * d.x);
        } else if (h == 1) {  // + i ky F(v f)
          v[j] = make_double2(fma(-ky, d.y, v[j].x), fma(ky, d.x, v[j].y));
        } else {
          v[j] = make_double2(v[j].x + d.x, v[j].y + d.y);
        }
      }
    });
  }
  sfor<R>([&](auto jj) {
    constexpr int j = decltype(jj)::value;
    const int r = l < L ? kept_row(k, pos_row<N>(k, l + L * j)) : -1;
    if (r >= 0 && live) tile[(size_t)r * TS + cc] = v[j];
  });
  __syncthreads();
  double2* out = (f == 0) ? k.Aq : (f == 1 ? k.Aw : k.Ath);
  for (int i = threadIdx.x; i < k.Mr * CB; i += blockDim.x) {
    const int r = i / CB, cc2 = i % CB;
    if (cc2 >= ncb) continue;
    const int c2 = c0 + cc2;
    const size_t o = k.full_out
                         ? ((size_t)lev * k.Nx + full_row(r, k.K, k.Mr, k.Nx)) * k.Nk + c2
                         : (size_t)lev * k.M + (size_t)r * k.Mc + c2;
    out[o] = tile[(size_t)r * TS + cc2];
  }
}

// H1's CTAs take one raw field or two, H3's one output field: splitting them
// over fields repeats nothing and shortens the last wave (256^2 x 33 levels:
// H1 84 -> 73 us, H3 162 -> 125; at 257 levels equal).  H2 split over the
// output fields transforms the velocity factors in each of the three CTAs, and
// H1 stages less at a time with one field than with two, so these two are taken
// only while the pieces leave the chip half empty, 8 of 16 warps an SM (H2 at
// 64^2 x 49 levels 34.8 -> 22.5 us; at 64^2 x 97 and 96^2 x 49, the next above
// the line, 39.5 -> 40.9 and 83 -> 86).
constexpr int kSplitWarps = 152 * 8;

template <int R, int L, int P, int Q>
cudaError_t launch(const HX& args, cudaStream_t st, Profiler& prof) {
  HX k = args;
  using F = Lane<R, L, P, Q>;
  constexpr int N = F::N, CB = F::CB;
  const size_t head = head_bytes<F>();
  const size_t field = (size_t)k.rows_in * (CB + 1) * sizeof(double2);
  const int c1 = (k.cols_in + CB - 1) / CB, c2 = (N / 2 + CB - 1) / CB, c3 = (k.Mc + CB - 1) / CB;
  k.stage = head + 2 * field <= 112 * 1024 && 4 * c1 * k.levels * F::W > kSplitWarps ? 2 : 1;
  const int h2z = 3 * c2 * k.levels * F::W <= kSplitWarps ? 3 : 1;
  const size_t sm1 = head + k.stage * field;
  const size_t sm2 = head + (size_t)CB * 2 * R * F::LS * sizeof(cfx);
  const size_t sm3 = head + (size_t)k.Mr * (CB + 1) * sizeof(double2);
  auto h2 = k_h2x<F, HF_JAC, false>;
  if (k.form == HF_FLUX) h2 = k.sponge ? k_h2x<F, HF_FLUX, true> : k_h2x<F, HF_FLUX, false>;
  prof.begin("h1_col_ifft", st);
  launch_after(k_h1x<F>, dim3(c1, k.levels, 4 / k.stage), 32 * F::W, sm1, st, k);
  prof.end(st);
  prof.begin("h2_row_products", st);
  launch_after(h2, dim3(c2, k.levels, h2z), 32 * F::W, sm2, st, k);
  prof.end(st);
  prof.begin("h3_col_fft", st);
  launch_after(k_h3x<F>, dim3(c3, k.levels, 3), 32 * F::W, sm3, st, k);
  prof.end(st);
  return cudaGetLastError();
}

}  // namespace hfx
}  // namespace nhqg
