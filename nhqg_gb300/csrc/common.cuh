// Shared device helpers for the NHQG GB300 engine (FP64 plain path).
//
// Complex values are double2 (x = re, y = im).  On GB300 the FP64 pipe
// retires ~2 DFMA/clk/SM, ~58x fewer lanes than FP32, so every kernel here
// is written to minimise FP64 instructions; integer/shared-memory work is
// close to free next to it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace nhqg {

// Programmatic dependent launch.  A step is a chain of kernels, and at small
// sizes the gaps between them weigh as much as the kernels: launch_after() hands
// the next grid to the GPU before the previous one has ended, and its CTAs,
// which start as the previous grid's leave, wait in after_previous() (all of that
// grid done, its writes visible) before they touch anything a kernel writes.
// Every CTA of every kernel launched that way calls it, so completion stays ordered
// along the stream.  Before it a kernel may read constant tables, and what a kernel
// before the previous one left: its CTAs start when every CTA of the previous grid has
// exited, each of which had waited for the grid before that.  k_corr_tstep alone does the
// latter (run_corrector states the order it needs).  Per step: 64^2 x 32 plain 661
// -> 570 us, 96^2 x 48 mixed 600 -> 520.  Letting the next grid in early
// (launch_dependents at the start of each kernel) measured 726 and 665: its
// waiting CTAs take the SMs' slots.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Lets a kernel take `bytes` of dynamic shared memory.  The limit belongs to the
// function, not to the launch: setting it to each launch's own size let a thread with
// a smaller launch of the same kernel lower it between another's call and launch,
// which then failed.  It is only ever set to one of two values that cover the launch,
// 200 KB, or all that the kernel's static shared memory leaves.
template <typename... P>
inline cudaError_t allow_smem(void (*kern)(P...), size_t bytes) {
  if (bytes <= 32 * 1024) return cudaSuccess;  // within the default 48 KB, static part included
  int lim = 200 * 1024;
  if (bytes > (size_t)lim) {
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, kern);
    if (e != cudaSuccess) return e;
    lim = 227 * 1024 - (int)fa.sharedSizeBytes;
  }
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
}

template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                A&&... args) {
  const cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, std::forward<A>(args)...);
}

__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
// i * a
__device__ __forceinline__ double2 cmul_i(double2 a) { return make_double2(-a.y, a.x); }
// a * b
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
// acc + s * a  (s real)
__device__ __forceinline__ double2 caxpy(double s, double2 a, double2 acc) {
  return make_double2(fma(s, a.x, acc.x), fma(s, a.y, acc.y));
}
__device__ __forceinline__ double2 czero() { return make_double2(0.0, 0.0); }

// Sizes of one grid.  Compact mode layout: the stored modes are Mr rows in
// fftfreq order (kx_int = 0..K, then the Mr-K-1 most negative rows) times Mc
// columns ky = 0..Mc-1; mode m = r*Mc + c; a field is [level][m].
//  - 2/3 rule: the keep-rectangle |kx_int| <= K, ky_int <= K with K = Nx/3,
//    Mr = 2K+1, Mc = K+1; products are formed on the Nx grid (Nh = Nx).
//  - 3/2 rule: every rfft2 mode (the state is full band): K = Nx/2 (the
//    Nyquist row counts as a "positive" row), Mr = Nx, Mc = Nk; products are
//    formed on the zero-padded Npad = 3Nx/2 grid (Nh = Npad).
struct Dims {
  int Nx, Nk, Nz, P, G, K, Mr, Mc, M;
  int Nh;    // side of the physical grid the horizontal products use
  bool pad;  // 3/2 rule (full-band layout, padded products)
};

inline Dims make_dims(int Nx, int Nz, bool pad32 = false) {
  Dims d;
  d.Nx = Nx;
  d.Nk = Nx / 2 + 1;
  d.Nz = Nz;
  d.P = Nz + 1;
  d.G = Nz - 1;
  d.pad = pad32;
  if (pad32) {
    d.K = Nx / 2;
    d.Mr = Nx;
    d.Mc = d.Nk;
    d.Nh = 3 * Nx / 2;
  } else {
    d.K = Nx / 3;
    d.Mr = 2 * d.K + 1;
    d.Mc = d.K + 1;
    d.Nh = Nx;
  }
  d.M = d.Mr * d.Mc;
  return d;
}

// full-layout kx row of compact row r
__host__ __device__ __forceinline__ int full_row(int r, int K, int Mr, int Nx) {
  return r <= K ? r : Nx - Mr + r;
}
// compact row of the mirrored wavenumber -kx (ky = 0 column pairing; the
// Nyquist row of the full-band layout is its own mirror)
__host__ __device__ __forceinline__ int mirror_row(int r, int Mr) {
  return r == 0 ? 0 : Mr - r;
}
// row of the zero-padded Nh-point spectrum that holds full-layout row kf
// (nhqg/spectral.py:18-34: rows 0..Nx/2-1 stay, rows Nx/2..Nx-1 move to the
// top, so the Nyquist row becomes kx = -Nx/2); the identity when Nh == Nx
__host__ __device__ __forceinline__ int padded_row(int kf, int Nx, int Nh) {
  return kf < Nx / 2 ? kf : kf + (Nh - Nx);
}

// Block-wide deterministic sum of one double per thread (blockDim <= 1024).
__device__ __forceinline__ double block_sum(double v, double* scratch) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  double t = 0.0;
  if (warp == 0) {
    t = lane < nw ? scratch[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// Division by a number known at run time, n / d for 0 <= n, n d < 2^32, by one
// multiplication: m = ceil(2^32 / d) exceeds 2^32 / d by less than 1, so that
// the quotient's error stays below n / 2^32 < 1 / d.  The index arithmetic of the
// transforms' lengths with a factor 3 spent more instructions on divisions than
// on the transforms.
struct Div {
  int d;
  unsigned m;
  __host__ __device__ static unsigned magic(int d) { return d > 1 ? 0xffffffffu / (unsigned)d + 1u : 0u; }
  __device__ __forceinline__ explicit Div(int d_) : d(d_), m(magic(d_)) {}
  __device__ __forceinline__ Div(int d_, unsigned m_) : d(d_), m(m_) {}  // m = magic(d)
  // n / d; r = n % d
  __device__ __forceinline__ int operator()(int n, int& r) const {
    const int q = d > 1 ? (int)__umulhi((unsigned)n, m) : n;
    r = n - q * d;
    return q;
  }
};

}  // namespace nhqg
