// Host side of the fixed-point horizontal products (horizontal_fx.cuh): tables,
// the rule that takes a call to them, and the dispatch over lengths.
#include <cmath>

#include "horizontal_fx.cuh"

namespace nhqg {

cudaError_t launch_hfx_48(const hfx::HX&, cudaStream_t, Profiler&);
cudaError_t launch_hfx_64(const hfx::HX&, cudaStream_t, Profiler&);
cudaError_t launch_hfx_72(const hfx::HX&, cudaStream_t, Profiler&);
cudaError_t launch_hfx_96(const hfx::HX&, cudaStream_t, Profiler&);
cudaError_t launch_hfx_128(const hfx::HX&, cudaStream_t, Profiler&);
cudaError_t launch_hfx_144(const hfx::HX&, cudaStream_t, Profiler&);
cudaError_t launch_hfx_192(const hfx::HX&, cudaStream_t, Profiler&);
cudaError_t launch_hfx_256(const hfx::HX&, cudaStream_t, Profiler&);

// Lengths R L in three register stages (hfx::Lane), at most 32 lanes of 8 or 12 values;
// others (longer ones, and the tiny test grids) keep the FP64 kernels of
// horizontal.cu.
bool horizontal_fx_supported(int N) {
  switch (N) {
    case 48: case 64: case 72: case 96: case 128: case 144: case 192: case 256: return true;
    default: return false;
  }
}

// exp(+2 pi i k / N), k < n <= N, in units 2^-61
std::vector<fx::cfx> fx_roots(int n, int N) {
  std::vector<fx::cfx> out(n);
  const long double pi4 = 0.785398163397448309615660845819875721L;
  const long double one = std::ldexp(1.0L, fx::kBits);
  for (int k = 0; k < n; ++k) {
    // octant reduction: the angle handed to cosl / sinl lies in [0, pi/4]
    const int k8 = 8 * k, oct = k8 / N;
    int r = k8 - oct * N;
    if (oct & 1) r = N - r;
    const long double a = pi4 * r / N;
    const long long c = std::llround(std::cos(a) * one), s = std::llround(std::sin(a) * one);
    const long long cs[8] = {c, s, -s, -c, -c, -s, s, c}, sn[8] = {s, c, c, s, -s, -c, -c, -s};
    out[k] = fx::cfx{cs[oct], sn[oct]};
  }
  return out;
}

// exp(+2 pi i k / N), k < N, as the 6 integers of fx::Tw
std::vector<int> horizontal_fx_twiddles(int N) {
  std::vector<int> out;
  for (const fx::cfx& r : fx_roots(N, N)) {
    const fx::Tw w = fx::make_tw(r.x, r.y);
    for (int v : {w.ch, w.cl, w.dh, w.dl, w.nh, w.nl}) out.push_back(v);
  }
  return out;
}

// v * s as integers, each run of `run` values at one exponent above every |v s|;
// a run with an infinity or a NaN gets kENan
void horizontal_fx_table(const std::vector<double>& v, double s, size_t run, std::vector<long long>& out,
                         std::vector<int>& e) {
  out.resize(v.size());
  e.assign(v.size() / run, -900);
  for (size_t b = 0; b < e.size(); ++b) {
    double m = 0.0;
    bool finite = true;
    for (size_t i = b * run; i < (b + 1) * run; ++i) {
      finite = finite && std::isfinite(v[i] * s);
      m = std::max(m, std::fabs(v[i] * s));
    }
    if (!finite) e[b] = fx::kENan;
    else if (m > 0.0) std::frexp(m, &e[b]);
    e[b] += 1;
    for (size_t i = b * run; i < (b + 1) * run; ++i) out[i] = fx::to_fx(v[i] * s, e[b]);
  }
}

// The fixed-point kernels take the flux and Jacobian forms at their lengths
// where the context holds their tables; the Jacobian with a sponge (11 input
// fields) and the sponge-only product stay with the FP64 kernels.
bool horizontal_fx_takes(const Params& p, const Tables& t, const Work& w, const HorizArgs& a) {
  if (!t.fx.tw || !w.e1 || !horizontal_fx_supported(p.d.Nh)) return false;
  if (a.form == HF_FLUX) return !a.sponge || t.fx.sponge != nullptr;
  return a.form == HF_JAC && !a.sponge;
}

cudaError_t launch_horizontal_fx(const Params& p, const Tables& t, Work& w, const HorizArgs& a,
                                 cudaStream_t st, int* nlaunch) {
  const Dims& d = p.d;
  hfx::HX k{};
  k.Nx = d.Nx; k.Nk = d.Nk; k.K = d.K; k.Mr = d.Mr; k.Mc = d.Mc; k.M = d.M;
  k.levels = a.levels;
  k.full_in = a.full_in;
  k.full_out = a.full_out;
  k.rows_in = a.full_in ? d.Nx : d.Mr;
  k.cols_in = a.full_in ? d.Nk : d.Mc;
  k.form = a.form;
  k.sponge = a.sponge;
  k.eta = a.eta;
  k.psi_derived = a.psi_derived;
  k.nf1 = a.form == HF_FLUX ? 5 : 8;
  k.ng = a.form == HF_FLUX ? (a.sponge ? 9 : 6) : 3;
  k.psi = a.psi; k.q = a.q; k.w = a.w; k.th = a.th;
  k.kx = t.kx_full; k.ky = t.ky_full;
  k.kx_s = t.fx.kx_s; k.ky_s = t.fx.ky_s;
  k.inv_denom = t.inv_denom;
  k.eta_c = t.eta;
  k.sponge_fx = t.fx.sponge; k.eta_fx = t.fx.eta;
  k.sponge_e = t.fx.sponge_e; k.eta_e = t.fx.eta_e;
  k.tw = t.fx.tw;
  k.Aq = a.Aq; k.Aw = a.Aw; k.Ath = a.Ath;
  if ((size_t)k.nf1 * a.levels * k.cols_in * d.Nh > w.x1_elems ||
      (size_t)k.ng * a.levels * d.Mc * d.Nh > w.x2_elems)
    return cudaErrorInvalidValue;
  k.x1 = reinterpret_cast<fx::cfx*>(w.x1);
  k.x2 = reinterpret_cast<fx::cfx*>(w.x2);
  k.e1 = w.e1;
  k.e2 = w.e2;
  if (nlaunch) *nlaunch += 3;
  switch (d.Nh) {
    case 48: return launch_hfx_48(k, st, w.prof);
    case 64: return launch_hfx_64(k, st, w.prof);
    case 72: return launch_hfx_72(k, st, w.prof);
    case 96: return launch_hfx_96(k, st, w.prof);
    case 128: return launch_hfx_128(k, st, w.prof);
    case 144: return launch_hfx_144(k, st, w.prof);
    case 192: return launch_hfx_192(k, st, w.prof);
    case 256: return launch_hfx_256(k, st, w.prof);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace nhqg
