// The per-rung smoothing: cuFFT R2C of the density contrast once, then per
// radius one fused filter kernel and a cuFFT C2R -- or, for the float form on
// a 512^3 grid (below) and the FP64 form on 128^3 and 256^3 (fft64.cu), three
// passes of its own that fuse the filter into the first.
//
// Replaces sif__fft_grid_forward, fft_build_filter_lut,
// sif__fft_apply_filter_smoothed and sif__fft_grid_backward
// (src/math/fft.c:790-818, 521-568, 703-788, 820-888) and the window setup of
// sif__finder_deconvolve_window (src/finder/utils.c:75-110,
// src/math/fft.c:958-1046). cuFFT stands in for FFTW's planes and pencils.
//
// The filter kernel multiplies each mode by W(k R) (top-hat
// 3(sin x - x cos x)/x^3, or Gaussian exp(-x^2/2)), by the CIC window
// correction 1/sinc^2 per axis (or the aliasing-aware W/S), and by the C2R's
// 1/N^3, reading the spectrum once and writing the transform's input once.
// The radial factor comes from a table indexed by the integer |k|^2, built in
// double by a small kernel, as the reference tabulates it (the own inverse at
// 512 evaluates the same formulas in float as it applies them). The unfiltered
// pass (the grid handed back at the end of a run) applies no window, as the
// reference's SIF__FILTER_NONE copies the spectrum untouched.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "smooth.cuh"

namespace sifg {

#define SIFG_CUFFT(call)                                                        \
  do {                                                                          \
    cufftResult r_ = (call);                                                    \
    if (r_ != CUFFT_SUCCESS) throw ::sifg::CudaError{cudaErrorUnknown, #call};  \
  } while (0)

// The factor is even in kx and ky, so a thread finds it once, at (|kx|, |ky|,
// kz), and applies it to the up to four modes that share it: the table by
// |k|^2 is a gather whose lanes fall in as many cache lines, and with a gather
// a mode it was what the kernel waited on. (256^3: 33 us a pass of 135 MB with
// a gather a mode, 105 in double, where four products a mode cost more than
// the modes' own two.) Product by product the factor is the one a mode alone
// would have found.
template <class R>
struct Mode;
template <>
struct Mode<float> {
  using T = float2;
};
template <>
struct Mode<double> {
  using T = double2;
};

template <class R>
__global__ void __launch_bounds__(256) filter_kernel(const typename Mode<R>::T* __restrict__ spec,
                                                     typename Mode<R>::T* __restrict__ out, uint32_t n,
                                                     const R* __restrict__ lut,
                                                     const R* __restrict__ win, R norm) {
  using M = typename Mode<R>::T;
  const uint32_t zd = n / 2 + 1, half = n / 2 + 1;  // |k| from 0 to n / 2 on every axis
  const uint32_t ix = blockIdx.y, jx = ix == 0 || 2 * ix == n ? ix : n - ix;
  const R wx = win ? __ldg(win + ix) : R(1);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < half * zd; t += gridDim.x * blockDim.x) {
    const uint32_t iy = t / zd, iz = t - iy * zd;
    const uint32_t jy = iy == 0 || 2 * iy == n ? iy : n - iy;
    const size_t at[4] = {(size_t)(ix * n + iy) * zd + iz, (size_t)(ix * n + jy) * zd + iz,
                          (size_t)(jx * n + iy) * zd + iz, (size_t)(jx * n + jy) * zd + iz};
    const bool on[4] = {true, jy != iy, jx != ix, jx != ix && jy != iy};
    M v[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (on[k]) v[k] = __ldg(spec + at[k]);
    R s = __ldg(lut + (ix * ix + iy * iy + iz * iz)) * norm;
    if (win) s = s * wx * __ldg(win + iy) * __ldg(win + iz);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (!on[k]) continue;
      M o;
      o.x = v[k].x * s;
      o.y = v[k].y * s;
      out[at[k]] = o;
    }
  }
}

// ---------------------------------------------------------------------------
// The float form's inverse transform at n = 512, in three passes of its own
// in place of the filter kernel and cuFFT's C2R:
//   (1) filter + inverse FFT along kx (spectrum -> work),
//   (2) inverse FFT along ky (work, in place),
//   (3) C2R along kz (work -> the real grid).
// A 512-point transform belongs to 32 threads, 16 values each: a 16-point DFT
// in registers over the thread's stride-32 values, a twiddle, an exchange
// through shared memory, a second 16-point DFT and a radix-2 step between
// pairs of lanes by shuffles (512 = 16 x 32, 32 = 16 x 2). Passes (1) and (2)
// give a CTA 16 neighbouring kz columns of one line (128 contiguous bytes
// per row of the line); pass (3) gives each 257-mode kz row to a half-warp
// as a 256-point complex transform of the packed even and odd samples.
// Twiddles come from tables computed in double; the three passes read and
// write the transform's data once each.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul_i(float2 a) { return make_float2(-a.y, a.x); }  // a * i

// e^{+2 pi i k/32}, k < 16, rounded to float.
__constant__ float2 kW32[16] = {
    {1.0f, 0.0f},
    {0.9807852506637573f, 0.19509032368659973f},
    {0.9238795042037964f, 0.3826834261417389f},
    {0.8314695954322815f, 0.5555702447891235f},
    {0.7071067690849304f, 0.7071067690849304f},
    {0.5555702447891235f, 0.8314695954322815f},
    {0.3826834261417389f, 0.9238795042037964f},
    {0.19509032368659973f, 0.9807852506637573f},
    {0.0f, 1.0f},
    {-0.19509032368659973f, 0.9807852506637573f},
    {-0.3826834261417389f, 0.9238795042037964f},
    {-0.5555702447891235f, 0.8314695954322815f},
    {-0.7071067690849304f, 0.7071067690849304f},
    {-0.8314695954322815f, 0.5555702447891235f},
    {-0.9238795042037964f, 0.3826834261417389f},
    {-0.9807852506637573f, 0.19509032368659973f},
};

// Inverse (e^{+2 pi i jk/R}) DFTs of 4, 8 and 16 points, in place, natural order.
__device__ __forceinline__ void dft_inv(float2 (&v)[4]) {
  const float2 c0 = cadd(v[0], v[2]), c2 = csub(v[0], v[2]);
  const float2 c1 = cadd(v[1], v[3]), d = cmul_i(csub(v[1], v[3]));
  v[0] = cadd(c0, c1);
  v[2] = csub(c0, c1);
  v[1] = cadd(c2, d);
  v[3] = csub(c2, d);
}
__device__ __forceinline__ void dft_inv(float2 (&v)[8]) {
  const float h = 0.70710678118654752440f;  // cos(pi/4)
  float2 a[4], b[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    a[j] = cadd(v[j], v[j + 4]);
    b[j] = csub(v[j], v[j + 4]);
  }
  // b[j] *= w^j, w = e^{+i pi/4}
  b[1] = make_float2(h * (b[1].x - b[1].y), h * (b[1].x + b[1].y));
  b[2] = cmul_i(b[2]);
  b[3] = make_float2(-h * (b[3].x + b[3].y), h * (b[3].x - b[3].y));
  dft_inv(a);
  dft_inv(b);
#pragma unroll
  for (int m = 0; m < 4; m++) {
    v[2 * m] = a[m];
    v[2 * m + 1] = b[m];
  }
}
__device__ __forceinline__ void dft_inv(float2 (&v)[16]) {
  float2 e[8], o[8];
#pragma unroll
  for (int m = 0; m < 8; m++) {
    e[m] = v[2 * m];
    o[m] = v[2 * m + 1];
  }
  dft_inv(e);
  dft_inv(o);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    float2 t;
    if (k == 0)
      t = o[0];
    else if (k == 4)
      t = cmul_i(o[4]);
    else
      t = cmul(o[k], kW32[2 * k]);
    v[k] = cadd(e[k], t);
    v[k + 8] = csub(e[k], t);
  }
}

constexpr int kColCols = 16;

// Twiddle tables of the n = 512 transform, one device block:
//   [0, 512):    W512^(j k), at k * 32 + j (j < 32, k < 16), the column pass
//   [512, 768):  W256^(j k), at k * 16 + j (j, k < 16), the row pass
//   [768, 1024): W512^k, k < 256, the row pass's even/odd packing
constexpr int kTw512 = 1024;

// The filter of one kx column at (ky, kz): mode kx is scaled by
// lut[k^2] * norm * win[kx] * win[ky] * win[kz] (win optional), the factor
// and the order of its products as the per-mode filter kernel has them.
// The radial factor of the filter pass, evaluated where it is applied: a
// table by |k|^2 (as the other grids use) is a gather whose lanes fall in as
// many cache lines, and it doubled the pass's time. These are the table's
// formulas (fft_build_filter_lut, src/math/fft.c:521-568) in float: the
// top-hat 3 (sin x - x cos x) / x^3 by its Taylor series below x = 2, where
// the formula cancels, and through sin and cos above; the Gaussian
// exp(-x^2 / 2); the extra Gaussian of sigma on top of either. Above x = 2
// the phase x = f |k| carries its rounding error as a second float (f's low
// part, the square root's residual, the product's error by fma): a float x
// alone is off by up to x ulp, as much as 4e-6 in the factor at x = 70. sin
// and cos of that pair come from a reduction by pi/2 (Cody and Waite: pi/2 in
// three parts, the first two of 12 significant bits so that n times them is
// exact, the pair's low part added to the remainder) and Taylor series on
// [-pi/4, pi/4] (to x^9 and x^10: the first term left out is below 2e-10);
// within 1.5 ulp. The factor is then within about 4 ulp of the table's
// double value (2e-7 rms relative over the modes above x = 2).
struct RadialFilter {
  int kind;         // kFilterTopHat, kFilterGaussian, else 1
  float x2;         // x^2 per unit |k|^2: f^2, f = R 2 pi / L
  float g2;         // the extra Gaussian's exponent per unit |k|^2: (sigma 2 pi / L)^2 / 2; 0 for none
  float f, f_lo;    // f as a float and its remainder
};

// sin and cos of x + x_lo (|x_lo| below an ulp of x, 0 < x < 4096 pi / 2).
__device__ __forceinline__ void sincos_pair(float x, float x_lo, float& s, float& c) {
  constexpr float kP1 = 1.57080078125f;             // pi/2 to 12 bits
  constexpr float kP2 = -4.4535845518112183e-06f;   // the remainder to 12 bits
  constexpr float kP3 = (float)(1.57079632679489661923 - 1.57080078125 + 4.4535845518112183e-06);
  const float n = rintf(x * (float)(2.0 / 3.14159265358979323846));
  float r = fmaf(-n, kP1, x);  // exact: n kP1 has 24 bits and lies within a factor 2 of x
  r = fmaf(-n, kP2, r);
  r = fmaf(-n, kP3, r) + x_lo;
  const float r2 = r * r;
  float ps = (float)(1.0 / 362880.0);
  ps = fmaf(ps, r2, (float)(-1.0 / 5040.0));
  ps = fmaf(ps, r2, (float)(1.0 / 120.0));
  ps = fmaf(ps, r2, (float)(-1.0 / 6.0));
  const float sr = fmaf(ps * r2, r, r);
  float pc = (float)(-1.0 / 3628800.0);
  pc = fmaf(pc, r2, (float)(1.0 / 40320.0));
  pc = fmaf(pc, r2, (float)(-1.0 / 720.0));
  pc = fmaf(pc, r2, (float)(1.0 / 24.0));
  pc = fmaf(pc, r2, -0.5f);
  const float cr = fmaf(pc, r2, 1.0f);
  // x = n pi/2 + r: quadrant q of n turns (sin r, cos r) by q quarter turns.
  const int q = (int)n & 3;
  s = (q & 1) ? cr : sr;
  c = (q & 1) ? sr : cr;
  if (q & 2) s = -s;
  if ((q + 1) & 2) c = -c;
}

// The series sum_{n >= 1} (-1)^(n+1) 6n x^(2n-2) / (2n+1)! of the top-hat,
// through n = 8: the first term left out is below 3e-11 for x < 2.
__device__ __forceinline__ float tophat_series(float x2) {
  float p = (float)(-48.0 / 355687428096000.0);
  p = fmaf(p, x2, (float)(42.0 / 1307674368000.0));
  p = fmaf(p, x2, (float)(-36.0 / 6227020800.0));
  p = fmaf(p, x2, (float)(30.0 / 39916800.0));
  p = fmaf(p, x2, (float)(-24.0 / 362880.0));
  p = fmaf(p, x2, (float)(18.0 / 5040.0));
  p = fmaf(p, x2, (float)(-12.0 / 120.0));
  return fmaf(p, x2, 1.0f);
}

__device__ __forceinline__ float radial_factor(uint32_t k2, const RadialFilter& rf) {
  if (k2 == 0) return 1.0f;
  const float kk = (float)k2;  // exact: k2 <= 3 * 256^2
  float v = 1.0f;
  if (rf.kind == kFilterTopHat) {
    const float x2 = rf.x2 * kk;
    if (x2 < 4.0f) {
      v = tophat_series(x2);
    } else {
      // |k| as k + k_lo: a reciprocal square root, and the residual's
      // first-order correction (exact to well below an ulp whatever the
      // reciprocal's own error).
      const float y = rsqrtf(kk);
      const float k = kk * y;
      const float k_lo = fmaf(-k, k, kk) * (0.5f * y);
      const float x = rf.f * k;
      const float x_lo = fmaf(rf.f, k, -x) + fmaf(rf.f, k_lo, rf.f_lo * k);
      float s, c;
      sincos_pair(x, x_lo, s, c);
      v = 3.0f * fmaf(-x, c, s) * __frcp_rn(x2 * x);
    }
  } else if (rf.kind == kFilterGaussian) {
    v = expf(-0.5f * (rf.x2 * kk));
  }
  if (rf.g2 > 0.0f) v *= expf(-(rf.g2 * kk));
  return v;
}

constexpr RadialFilter kNoFilter{-1, 0.0f, 0.0f, 0.0f, 0.0f};  // a pass that applies no filter

// The factor table of a smoothing at n = 512: entry ((|ky| * 257 + |kx|) * 257
// + kz) holds the factor the filter pass applies to mode (kx, ky, kz) --
// radial_factor(k^2) * norm, then the window's three factors, in the order
// and with the values the pass computes them without the table, so the table
// changes no bit of the transform. kz runs fastest: the pass's lanes hold
// neighbouring kz.
constexpr uint32_t kFactorSide = 257;
__global__ void factor_table_kernel(float* __restrict__ tab, RadialFilter rf,
                                    const float* __restrict__ win, float norm) {
  constexpr uint64_t total = (uint64_t)kFactorSide * kFactorSide * kFactorSide;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t kz = (uint32_t)(i % kFactorSide);
    const uint32_t kx = (uint32_t)((i / kFactorSide) % kFactorSide);
    const uint32_t ky = (uint32_t)(i / ((uint64_t)kFactorSide * kFactorSide));
    float v = radial_factor(kx * kx + (ky * ky + kz * kz), rf) * norm;
    if (win) v = v * __ldg(win + kx) * __ldg(win + ky) * __ldg(win + kz);
    tab[i] = v;
  }
}

// The work buffer between the passes holds the half spectrum in tiles of 16
// kz columns by 512: tile (x, kb) holds kz = 16 kb .. 16 kb + 15 for every
// ky, at ((x * kKzBlocks + kb) * 512 + ky) * 16 + kz % 16. Pass (2) reads
// and writes each tile as one contiguous 64 KB block, pass (3) reads each
// row's modes as 16-row, 2 KB blocks. kz past 256 are never written or read.
constexpr uint32_t kKzBlocks = 17;
constexpr size_t kTileWorkElems = (size_t)512 * kKzBlocks * 512 * 16;

// Where passes (1) and (2) find their columns: element a of column kz of a
// line at line * line + kz / 16 * kblock + a * elem + kz % 16.
struct ColumnLayout {
  uint32_t line, kblock, elem;
};

// Passes (1) and (2), and the forward's ky and kx: the FFT along one axis of 16
// columns, 32 threads a column and 16 values a thread, neighbouring lanes on
// neighbouring kz. A thread loads its stride-32 values straight into registers
// and stores its results straight out, 128 contiguous bytes a half-warp either
// way; shared memory is crossed once, between the two 16-point stages, and the
// last radix-2 step goes between lanes 16 apart. A CTA takes one line's block of
// 16 kz; the columns of kz = 256, one a line, are taken 16 lines at a time by the
// last CTAs.
//
// Memory bounds it: 1.1 GB a pass at 512^3, 166 us at the measured copy rate.
// (With the tile staged through shared memory both ways, six crossings where
// this has two, and a warp a column: 215 us, 259 with the filter.)
//
// The filter (kColTable, kColEvaluate) scales each mode as it is read: by its
// entry in the smoothing's table, or by the factor evaluated. The forward DFT
// (e^{-2 pi i jk/512}) is the conjugate of the inverse DFT of the conjugate.
enum ColMode { kColInverse, kColForward, kColTable, kColEvaluate };
constexpr unsigned kColCtas = 512 * 16 + 512 / kColCols;
constexpr size_t kColBytes = (size_t)512 * kColCols * sizeof(float2);

template <ColMode kMode>
__global__ void __launch_bounds__(32 * kColCols, 2)
    colfft512_kernel(const float2* src, float2* dst, ColumnLayout in, ColumnLayout out,
                     const float2* __restrict__ tw, RadialFilter rf, const float* __restrict__ win,
                     float norm, const float* __restrict__ ftab, bool backwards) {
  extern __shared__ float2 ex[];  // element e of column c at e * kColCols + c
  const uint32_t c = threadIdx.x % kColCols, j = threadIdx.x / kColCols;
  // From the end backwards where the pass before went forwards within the same
  // planes: its last ones are still in L2 (the forward's ky after its rows: 186
  // to 174 us; the inverse's rows turned round after its ky 172 to 161).
  const uint32_t b = backwards ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const bool last = b >= 512 * 16;
  // The filter's lines in the order 0, 1, 511, 2, 510, ...: ky and -ky share the
  // table's entries, which are still in L2 for the second (read from memory
  // twice, 712 MB a pass and 234 us; 650 and 221).
  uint32_t line = last ? (b - 512 * 16) * kColCols + c : b / 16;
  if (kMode == kColTable && !last) line = (line & 1u) ? (line + 1) / 2 : (512 - line / 2) & 511u;
  const uint32_t kb = last ? 16 : b % 16, kz = last ? 256 : kb * 16 + c;
  float2 v[16];
  {
    const float2* p = src + (size_t)line * in.line + kb * in.kblock + (kz & 15u) + (size_t)j * in.elem;
    const size_t step = (size_t)32 * in.elem;
#pragma unroll
    for (int r = 0; r < 16; r++) v[r] = p[r * step];
  }
  if constexpr (kMode == kColForward) {
#pragma unroll
    for (int r = 0; r < 16; r++) v[r].y = -v[r].y;
  }
  if constexpr (kMode == kColTable || kMode == kColEvaluate) {
    const uint32_t aky = line > 256 ? 512 - line : line;
    const uint32_t q = aky * aky + kz * kz;
    const float* t = ftab + (size_t)aky * (kFactorSide * kFactorSide) + kz;
    const float wy = win ? __ldg(win + line) : 1.f, wz = win ? __ldg(win + kz) : 1.f;
#pragma unroll
    for (int r = 0; r < 16; r++) {
      const uint32_t kx = j + 32u * r, a = kx > 256 ? 512 - kx : kx;
      float s;
      if constexpr (kMode == kColTable) {
        s = __ldg(t + a * kFactorSide);
      } else {
        s = radial_factor(a * a + q, rf) * norm;
        if (win) s = s * __ldg(win + a) * wy * wz;
      }
      // Rounded as a product: fused into the transform's first sums it would
      // be other bits than a mode scaled and stored.
      v[r] = make_float2(__fmul_rn(v[r].x, s), __fmul_rn(v[r].y, s));
    }
  }
  dft_inv(v);
#pragma unroll
  for (int k = 1; k < 16; k++) v[k] = cmul(v[k], __ldg(tw + k * 32 + j));
#pragma unroll
  for (int k = 0; k < 16; k++) ex[(k * 32 + j) * kColCols + c] = v[k];
  __syncthreads();
  const uint32_t k1 = j >> 1, q = j & 1u;
#pragma unroll
  for (int m = 0; m < 16; m++) v[m] = ex[(k1 * 32 + q + 2 * m) * kColCols + c];
  dft_inv(v);  // E_q[k], k < 16
  // The radix-2 step between the two threads: X[k1 + 16 k] = E_0[k] + W32^k
  // E_1[k], X[k1 + 16 (k + 16)] = E_0[k] - W32^k E_1[k]. q = 0 finishes k < 8,
  // q = 1 k >= 8; each sends the half of its E it does not keep, and
  // W32^(8 + i) = i W32^i leaves one twiddle per register for both.
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float2 send = q ? v[i] : v[8 + i];
    const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, send.x, kColCols),
                                   __shfl_xor_sync(0xffffffffu, send.y, kColCols));
    const float2 a = q ? got : v[i];              // E_0[8 q + i]
    const float2 b = q ? cmul_i(v[8 + i]) : got;  // E_1[8 q + i] (times i for q = 1)
    const float2 t = i == 0 ? b : cmul(b, kW32[i]);
    v[i] = cadd(a, t);
    v[8 + i] = csub(a, t);
  }
  float2* p = dst + (size_t)line * out.line + kb * out.kblock + (kz & 15u) +
              (size_t)(k1 + 128 * q) * out.elem;
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const float2 o = kMode == kColForward ? make_float2(v[i].x, -v[i].y) : v[i];
    p[(size_t)(i < 8 ? 16 * i : 256 + 16 * (i - 8)) * out.elem] = o;
  }
}
static_assert(2 * kColCols == 32, "a column's thread pairs lie in one warp");

// Pass (3) and the forward's first: 16 rows per CTA, a half-warp a row, as a
// 256-point complex transform of the packed even and odd samples. A lane loads
// its values straight into registers and stores its results straight out, 128
// contiguous bytes a half-warp; shared memory is crossed once, between the two
// 16-point stages (slot 16 k1 + (j ^ k1) of the row), and the partner mode 256 -
// k comes by shuffle from the lane that holds it: value r of lane j is k = j +
// 16 r, so its partner is value 15 - r of lane 16 - j, and lane 0's its own
// value 16 - r.
//
// Memory bounds both: 1.1 GB each at 512^3, 166 us at the measured copy rate.
// (With the rows staged through shared memory both ways shared memory bound
// them: 187 us the inverse, 205 the forward.)
constexpr int kRowsPerCta = 16;
static_assert(kRowsPerCta * 512 == kBelowBlock, "a CTA's cells are one below-list block");

// The 256-point inverse DFT of a row, value r of lane j at j + 16 r before and
// after.
__device__ __forceinline__ void row256(float2 (&v)[16], float2* row, unsigned j,
                                       const float2* __restrict__ twb) {
  dft_inv(v);
#pragma unroll
  for (int k = 1; k < 16; k++) v[k] = cmul(v[k], __ldg(twb + k * 16 + j));
#pragma unroll
  for (int k = 0; k < 16; k++) row[16 * k + (j ^ k)] = v[k];
  __syncwarp();
#pragma unroll
  for (int m = 0; m < 16; m++) v[m] = row[16 * j + (m ^ j)];
  dft_inv(v);
}

// The partner of each value; `own0` is what lane 0's value 0 takes.
__device__ __forceinline__ void partners(const float2 (&z)[16], float2 own0, unsigned j,
                                         float2 (&m)[16]) {
#pragma unroll
  for (int r = 0; r < 16; r++) {
    m[r] = make_float2(__shfl_sync(0xffffffffu, z[15 - r].x, (16 - (int)j) & 15, 16),
                       __shfl_sync(0xffffffffu, z[15 - r].y, (16 - (int)j) & 15, 16));
    if (j == 0) m[r] = r == 0 ? own0 : z[(16 - r) & 15];
  }
}

// Pass (3). With Z the row's modes (the imaginary parts of Z[0] and Z[256]
// taken as zero, as a C2R does), c[k] = Fe[k] + i Fo[k] for k < 256, Fe = Z[k] +
// conj Z[256-k], Fo = (Z[k] - conj Z[256-k]) W512^k, and its inverse DFT y gives
// the real samples x[2m] = Re y[m], x[2m+1] = Im y[m].
//
// With `below` set the pass also lists, in flat order, the cells it writes
// whose value is at most below.thr: the CTA's 8192 cells are one contiguous
// flat range, and their entries go to the start of the CTA's own region of
// 8192 slots, their number to below.counts[CTA] (the candidate scan's
// threshold test, from the values in hand).
__global__ void __launch_bounds__(16 * kRowsPerCta, 3)
    c2r512_rows_kernel(const float2* __restrict__ work, float* __restrict__ out,
                       const float2* __restrict__ tw, BelowList below) {
  __shared__ float2 buf[kRowsPerCta * 256];
  // From the end backwards: the pass along ky, just before, left the last planes
  // it wrote in L2.
  const uint32_t block = gridDim.x - 1 - blockIdx.x;
  const uint32_t x = block / (512 / kRowsPerCta);
  const uint32_t y0 = (block % (512 / kRowsPerCta)) * kRowsPerCta;
  const unsigned j = threadIdx.x & 15u, ry = threadIdx.x >> 4;
  // The row's kz block 0; a kz block further is 512 rows of 16 on.
  const float2* p = work + ((size_t)x * kKzBlocks * 512 + y0 + ry) * 16 + j;
  constexpr size_t kBlock = (size_t)512 * 16;
  float2 v[16];
  {
    float2 z[16], zc[16], last = make_float2(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < 16; r++) z[r] = __ldg(p + r * kBlock);
    if (j == 0) {
      last = __ldg(p + 16 * kBlock);
      z[0].y = last.y = 0.f;
    }
    partners(z, last, j, zc);
    const float2* wpre = tw + 768;
#pragma unroll
    for (int r = 0; r < 16; r++) {
      const float2 c = make_float2(zc[r].x, -zc[r].y);
      const float2 fe = cadd(z[r], c), fo = cmul(csub(z[r], c), __ldg(wpre + j + 16u * r));
      v[r] = make_float2(fe.x - fo.y, fe.y + fo.x);
    }
  }
  row256(v, buf + ry * 256, j, tw + 512);
  float2* dst = reinterpret_cast<float2*>(out + ((size_t)x * 512 + y0 + ry) * 512) + j;
  if (!below.counts || below.field) {
#pragma unroll
    for (int k = 0; k < 16; k++) dst[16 * k] = v[k];
  }
  if (!below.counts) return;
  // Each lane's threshold bits, two a pair; the warps' totals place each
  // warp's entries (two rows, one after the other), each step of 16 pairs of
  // a row in lane order.
  constexpr uint32_t kWarps = 16 * kRowsPerCta / 32;
  __shared__ uint32_t ws[kWarps];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t bits = 0;
#pragma unroll
  for (int k = 0; k < 16; k++)
    bits |= ((v[k].x <= below.thr ? 1u : 0u) | (v[k].y <= below.thr ? 2u : 0u)) << (2 * k);
  const uint32_t n_mine = (uint32_t)__popc(bits);
  const uint32_t n_warp = __reduce_add_sync(0xffffffffu, n_mine);
  const uint32_t n_first = __reduce_add_sync(0xffffffffu, lane < 16 ? n_mine : 0u);
  if (lane == 0) ws[warp] = n_warp;
  __syncthreads();
  uint32_t pos = 0, total = 0;
#pragma unroll
  for (uint32_t w = 0; w < kWarps; w++) {
    pos += w < warp ? ws[w] : 0u;
    total += ws[w];
  }
  if (threadIdx.x == 0) below.counts[block] = total;
  if (n_warp == 0) return;
  const uint32_t row_lanes = lane < 16 ? 0xffffu : 0xffff0000u;
  const uint32_t lower = row_lanes & ((1u << lane) - 1u);
  if (lane >= 16) pos += n_first;
  const uint32_t cell0 = ((x * 512 + y0 + ry) * 512) + 2 * j;
  const size_t region = (size_t)block * (kRowsPerCta * 512);
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const uint32_t b = (bits >> (2 * k)) & 3u;
    const uint32_t mx = __ballot_sync(0xffffffffu, b & 1u), my = __ballot_sync(0xffffffffu, b & 2u);
    if ((mx | my) == 0u) continue;
    uint32_t at = pos + __popc(mx & lower) + __popc(my & lower);
    if (b & 1u) {
      below.delta[region + at] = v[k].x;
      below.flat[region + at] = cell0 + 32 * k;
      at++;
    }
    if (b & 2u) {
      below.delta[region + at] = v[k].y;
      below.flat[region + at] = cell0 + 32 * k + 1;
    }
    pos += __popc(mx & row_lanes) + __popc(my & row_lanes);
  }
}

// The forward transform's first pass, the R2C along z. The row read as 256
// complex values c[m] = x[2m] + i x[2m+1] is transformed forward (the conjugate
// of the inverse of the conjugate); then, with C[-k] taken mod 256, E[k] = (C[k]
// + conj C[-k]) / 2, O[k] = (C[k] - conj C[-k]) / 2i and X[k] = E[k] + W512^-k
// O[k] for k < 256, X[256] = E[0] - O[0]. The 257 modes go to the tiles.
__global__ void __launch_bounds__(16 * kRowsPerCta, 3)
    r2c512_rows_kernel(const float* __restrict__ grid, float2* __restrict__ work,
                       const float2* __restrict__ tw, const double* __restrict__ mean) {
  __shared__ float2 buf[kRowsPerCta * 256];
  const uint32_t x = blockIdx.x / (512 / kRowsPerCta);
  const uint32_t y0 = (blockIdx.x % (512 / kRowsPerCta)) * kRowsPerCta;
  const unsigned j = threadIdx.x & 15u, ry = threadIdx.x >> 4;
  const float2* src = reinterpret_cast<const float2*>(grid + ((size_t)x * 512 + y0 + ry) * 512) + j;
  float2 v[16];
#pragma unroll
  for (int r = 0; r < 16; r++) v[r] = __ldg(src + 16 * r);
  // With the mean, the rows are the density: its contrast, as the contrast
  // kernel computes it (inv rounded from the double 1 / mean), the double
  // division done once for the CTA while its loads land.
  if (mean) {
    __shared__ float inv_s;
    if (threadIdx.x == 0) inv_s = (float)(1.0 / __ldg(mean));
    __syncthreads();
    const float inv = inv_s;
#pragma unroll
    for (int r = 0; r < 16; r++)
      v[r] = make_float2(__fsub_rn(__fmul_rn(v[r].x, inv), 1.0f),
                         __fsub_rn(__fmul_rn(v[r].y, inv), 1.0f));
  }
#pragma unroll
  for (int r = 0; r < 16; r++) v[r].y = -v[r].y;
  row256(v, buf + ry * 256, j, tw + 512);
#pragma unroll
  for (int r = 0; r < 16; r++) v[r].y = -v[r].y;  // C
  float2 m[16];
  partners(v, v[0], j, m);
  const float2* wpre = tw + 768;
  float2* p = work + ((size_t)x * kKzBlocks * 512 + y0 + ry) * 16 + j;
  constexpr size_t kBlock = (size_t)512 * 16;
#pragma unroll
  for (int r = 0; r < 16; r++) {
    const float2 c = v[r];
    const float2 e = make_float2(0.5f * (c.x + m[r].x), 0.5f * (c.y - m[r].y));  // (C + conj C[-k]) / 2
    const float2 d = make_float2(c.x - m[r].x, c.y + m[r].y);                    // C - conj C[-k]
    const float2 o = make_float2(0.5f * d.y, -0.5f * d.x);                       // d / 2i
    const float2 w = __ldg(wpre + j + 16u * r);
    p[r * kBlock] = cadd(e, cmul(o, make_float2(w.x, -w.y)));
    if (r == 0 && j == 0) p[16 * kBlock] = make_float2(e.x - o.x, e.y - o.y);
  }
}

static bool own_inverse(uint32_t n) { return n == 512; }

// fft_build_filter_lut, src/math/fft.c:521-568: the radial factor by integer
// |k|^2, computed in double.
template <class R>
__device__ __forceinline__ R lut_value(uint32_t k2, int filter, double factor, double gfactor) {
  double v;
  if (k2 == 0) {
    v = 1.0;
  } else if (filter == kFilterTopHat) {
    const double kr = factor * sqrt((double)k2);
    v = kr > 1e-4 ? 3.0 * (sin(kr) - kr * cos(kr)) / (kr * kr * kr) : 1.0;
  } else if (filter == kFilterGaussian) {
    v = exp(-0.5 * factor * factor * (double)k2);
  } else {
    v = 1.0;
  }
  if (gfactor > 0.0 && k2 > 0) v *= exp(-0.5 * gfactor * gfactor * (double)k2);
  return (R)v;
}

// One table a blockIdx.y. A small grid's tables are built together, before its
// transform and beside its deposit: in line, each rung's smoothing waits for
// its own (double precision runs at a sixty-fourth of the float rate here: 7 us
// of a 64^3 smoothing's 35).
constexpr uint32_t kLutSet = 64;
struct LutSet {
  double factor[kLutSet], gfactor[kLutSet];
};
template <class R>
__global__ void lut_kernel(R* __restrict__ lut, uint32_t max_k2, int filter, LutSet set) {
  const double factor = set.factor[blockIdx.y], gfactor = set.gfactor[blockIdx.y];
  R* out = lut + (size_t)blockIdx.y * (max_k2 + 1);
  for (uint32_t k2 = blockIdx.x * blockDim.x + threadIdx.x; k2 <= max_k2;
       k2 += gridDim.x * blockDim.x)
    out[k2] = lut_value<R>(k2, filter, factor, gfactor);
}

template <class R>
SmootherT<R>::~SmootherT() {
  release();
}

template <class R>
static void destroy_plans(typename SmootherT<R>::Plans& p) {
  if (p.r2c) cufftDestroy(p.r2c);
  if (p.c2r) cufftDestroy(p.c2r);
  for (cufftHandle h : p.lane)
    if (h) cufftDestroy(h);
  if (p.twiddles) cudaFree(p.twiddles);
}

// A plan without a work area of its own (the smoother's shared one is set
// before it runs); `need` grows to the area it asks for.
static cufftHandle make_plan(uint32_t n, cufftType type, size_t* need) {
  cufftHandle h = 0;
  SIFG_CUFFT(cufftCreate(&h));
  size_t ws = 0;
  const cufftResult a = cufftSetAutoAllocation(h, 0);
  const cufftResult m = a == CUFFT_SUCCESS ? cufftMakePlan3d(h, (int)n, (int)n, (int)n, type, &ws) : a;
  if (m != CUFFT_SUCCESS) {
    cufftDestroy(h);
    throw CudaError{cudaErrorUnknown, "cufftMakePlan3d"};
  }
  if (ws > *need) *need = ws;
  return h;
}

template <class R>
void SmootherT<R>::release() {
  for (auto& p : plans) destroy_plans<R>(p);
  plans.clear();
  plan_r2c = plan_c2r = 0;
  plan_work = 0;
  twiddles = nullptr;
  factor_tables.clear();
  n = 0;
}

template <class R>
void SmootherT<R>::setup(uint32_t n_, R box_, int window_mode_, cudaStream_t st) {
  constexpr bool dbl = sizeof(R) == 8;
  bool rebind = false;
  if (n_ != n) {
    auto it = std::find_if(plans.begin(), plans.end(), [&](const Plans& p) { return p.n == n_; });
    if (it == plans.end()) {
      if ((int)plans.size() >= kPlanCache) {
        destroy_plans<R>(plans.front());
        plans.erase(plans.begin());
      }
      Plans p{n_, 0, 0};
      if (dbl && fft64_takes(n_)) {
        const std::vector<double> t = fft64_tables(n_);
        SIFG_CUDA(cudaMalloc(&p.twiddles, t.size() * sizeof(double)));
        SIFG_CUDA(cudaMemcpyAsync(p.twiddles, t.data(), t.size() * sizeof(double),
                                  cudaMemcpyHostToDevice, st));
        SIFG_CUDA(cudaStreamSynchronize(st));
      } else if (!dbl && own_inverse(n_)) {
        // The tables of the three-pass inverse, computed in double.
        std::vector<float2> tw(kTw512);
        auto root = [](double num, double den) {
          const double a = 2.0 * M_PI * num / den;
          return make_float2((float)std::cos(a), (float)std::sin(a));
        };
        for (int k = 0; k < 16; k++)
          for (int j = 0; j < 32; j++) tw[k * 32 + j] = root((double)(j * k), 512.0);
        for (int k = 0; k < 16; k++)
          for (int j = 0; j < 16; j++) tw[512 + k * 16 + j] = root((double)(j * k), 256.0);
        for (int k = 0; k < 256; k++) tw[768 + k] = root((double)k, 512.0);
        SIFG_CUDA(cudaMalloc(&p.twiddles, kTw512 * sizeof(float2)));
        // On the smoothing stream, which every use of the tables follows (a
        // plain cudaMemcpy runs on the legacy stream, which the library's
        // non-blocking streams do not wait for), and finished before the
        // staging vector goes.
        SIFG_CUDA(cudaMemcpyAsync(p.twiddles, tw.data(), kTw512 * sizeof(float2),
                                  cudaMemcpyHostToDevice, st));
        SIFG_CUDA(cudaStreamSynchronize(st));
      } else {
        p.r2c = make_plan(n_, dbl ? CUFFT_D2Z : CUFFT_R2C, &p.work);
        p.c2r = make_plan(n_, dbl ? CUFFT_Z2D : CUFFT_C2R, &p.work);
      }
      plans.push_back(p);
      it = plans.end() - 1;
    }
    n = n_;
    plan_r2c = it->r2c;
    plan_c2r = it->c2r;
    plan_work = it->work;
    twiddles = it->twiddles;
    rebind = true;  // a cached plan may be bound to another stream and area
  }
  if (plan_work > area.bytes) {
    area.ensure(plan_work);
    rebind = true;
  }
  if (rebind || st != stream) {
    for (cufftHandle h : {plan_r2c, plan_c2r}) {
      if (!h) continue;
      SIFG_CUFFT(cufftSetStream(h, st));
      if (plan_work) SIFG_CUFFT(cufftSetWorkArea(h, area.ptr));
    }
    stream = st;
  }
  box = box_;
  window_mode = window_mode_;
  const uint64_t modes = (uint64_t)n * n * (n / 2 + 1);
  spectrum.ensure(twiddles && !dbl ? kTileWorkElems * sizeof(float2) : modes * 2 * sizeof(R));
  work.ensure(twiddles && !dbl ? kTileWorkElems * sizeof(float2) : modes * 2 * sizeof(R));
  const uint32_t h = n >> 1;
  win.ensure((size_t)n * sizeof(R));
  if (window_mode) {
    // fft_build_window_axis, src/math/fft.c:958-975, CIC (order 2): 1/W full,
    // W/S aliasing-aware, W = sinc^2(pi k / N), S = 1 - 2 sin^2/3.
    std::vector<R> w(n);
    for (uint32_t i = 0; i < n; i++) {
      const int32_t k = i > h ? (int32_t)n - (int32_t)i : (int32_t)i;  // |k|: an even table
      const double x = M_PI * (double)k / (double)n;
      const double s = (x < 1e-9 && x > -1e-9) ? 1.0 : std::sin(x) / x;
      const double W = s * s;
      w[i] = (R)(window_mode == 2 ? W / (1.0 - 2.0 * std::sin(x) * std::sin(x) / 3.0) : 1.0 / W);
    }
    SIFG_CUDA(cudaMemcpyAsync(win.ptr, w.data(), n * sizeof(R), cudaMemcpyHostToDevice, st));
    SIFG_CUDA(cudaStreamSynchronize(st));
  }
}

template <class R>
uint32_t SmootherT<R>::lanes_for(uint32_t n_) const {
  if (sizeof(R) == 8 && fft64_takes(n_)) return kLanes;  // no plans
  for (const Plans& p : plans)
    if (p.n == n_) return std::min<uint32_t>(kLanes, 2 + (uint32_t)std::count_if(p.lane, p.lane + kLanes - 1,
                                                                               [](cufftHandle h) { return h != 0; }));
  return 1;
}

template <class R>
void SmootherT<R>::set_lanes(int lanes, const cudaStream_t* streams) {
  auto it = std::find_if(plans.begin(), plans.end(), [&](const Plans& p) { return p.n == n; });
  for (int k = 1; k < lanes; k++) {
    Lane& l = extra[k - 1];
    size_t need = plan_work;
    l.st = streams[k];
    l.work.ensure((uint64_t)n * n * (n / 2 + 1) * 2 * sizeof(R));
    if (twiddles) continue;  // no plans
    if (!it->lane[k - 1]) it->lane[k - 1] = make_plan(n, sizeof(R) == 8 ? CUFFT_Z2D : CUFFT_C2R, &need);
    if (need > it->work) it->work = need;
    l.c2r = it->lane[k - 1];
    SIFG_CUFFT(cufftSetStream(l.c2r, l.st));
    if (it->work) SIFG_CUFFT(cufftSetWorkArea(l.c2r, l.area.ensure(it->work)));
  }
}

template <class R>
const R* SmootherT<R>::tables(int filter, const R* radii, const R* sigmas, uint32_t count, DevBuf& buf,
                              cudaStream_t st) {
  const uint32_t h = n >> 1;
  const uint32_t max_k2 = 3 * h * h;
  R* out = (R*)buf.ensure((size_t)count * (max_k2 + 1) * sizeof(R));
  for (uint32_t k0 = 0; k0 < count; k0 += kLutSet) {
    const uint32_t nk = std::min(kLutSet, count - k0);
    LutSet set{};
    for (uint32_t k = 0; k < nk; k++) {
      set.factor[k] = (double)radii[k0 + k] * 2.0 * M_PI / (double)box;
      set.gfactor[k] = sigmas && sigmas[k0 + k] > R(0)
                           ? (double)sigmas[k0 + k] * 2.0 * M_PI / (double)box
                           : 0.0;
    }
    lut_kernel<R><<<dim3(grid_for((uint64_t)max_k2 + 1, 256), nk), 256, 0, st>>>(
        out + (size_t)k0 * (max_k2 + 1), max_k2, filter, set);
    SIFG_LAUNCH_CHECK();
  }
  return out;
}

static void launch_forward512(const SmootherT<float>& s, const float* grid, const double* mean);

template <>
void SmootherT<float>::forward(const float* grid, const double* mean) {
  if (twiddles) {
    launch_forward512(*this, grid, mean);
    return;
  }
  if (mean) apply_contrast(const_cast<float*>(grid), (uint64_t)n * n * n, mean, stream);
  SIFG_CUFFT(cufftExecR2C(plan_r2c, (cufftReal*)grid, (cufftComplex*)spectrum.ptr));
}
template <>
void SmootherT<double>::forward(const double* grid, const double* mean) {
  if (twiddles) {
    fft64_forward(n, grid, mean, spectrum.as<double2>(), (const double*)twiddles, stream);
    return;
  }
  if (mean) apply_contrast(const_cast<double*>(grid), (uint64_t)n * n * n, mean, stream);
  SIFG_CUFFT(cufftExecD2Z(plan_r2c, (cufftDoubleReal*)grid, (cufftDoubleComplex*)spectrum.ptr));
}

template <class R>
static void launch_filter(const SmootherT<R>& s, int filter, R norm, const R* lut, const DevBuf& work,
                          cudaStream_t st) {
  using M = typename Mode<R>::T;
  const R* w = (s.window_mode && filter != kFilterNone) ? s.win.template as<R>() : nullptr;
  const uint32_t half = s.n / 2 + 1;
  filter_kernel<R><<<dim3(grid_for((uint64_t)half * half, 256), half), 256, 0, st>>>(
      s.spectrum.template as<M>(), work.as<M>(), s.n, lut, w, norm);
}

// The three passes of the n = 512 inverse transform, on the smoother's stream.
// Tiles ((u * kKzBlocks + kb) * N + v) * 16 + kz % 16 read as columns along v
// with line u, or along u with line v. The forward leaves the spectrum as
// tiles of line ky along kx; the inverse's pass (1) writes the work buffer as
// tiles of line x along ky (read along x by nothing, along ky by pass (2)).
constexpr ColumnLayout kTilesByLine{kKzBlocks * 512 * kColCols, 512 * kColCols, kColCols};
constexpr ColumnLayout kTilesByRow{kColCols, 512 * kColCols, kKzBlocks * 512 * kColCols};

template <ColMode kMode>
static void launch_columns(const SmootherT<float>& s, const DevBuf& src, const DevBuf& dst,
                           ColumnLayout in, ColumnLayout out, const RadialFilter& rf = kNoFilter,
                           const float* win = nullptr, float norm = 1.f, const float* ftab = nullptr,
                           bool backwards = false) {
  thread_local bool attr = false;  // set once a thread: one device a process
  if (!attr) {
    SIFG_CUDA(cudaFuncSetAttribute(colfft512_kernel<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kColBytes));
    attr = true;
  }
  colfft512_kernel<kMode><<<kColCtas, 32 * kColCols, kColBytes, s.stream>>>(
      src.as<float2>(), dst.as<float2>(), in, out, (const float2*)s.twiddles, rf, win, norm, ftab,
      backwards);
  SIFG_LAUNCH_CHECK();
}

// The float form's forward transform at n = 512: the R2C along z into the
// work tiles, the forward ky FFT in place, the forward kx FFT into the
// spectrum's tiles.
static void launch_forward512(const SmootherT<float>& s, const float* grid, const double* mean) {
  constexpr uint32_t N = 512;
  r2c512_rows_kernel<<<N * N / kRowsPerCta, 16 * kRowsPerCta, 0, s.stream>>>(
      grid, s.work.as<float2>(), (const float2*)s.twiddles, mean);
  SIFG_LAUNCH_CHECK();
  launch_columns<kColForward>(s, s.work, s.work, kTilesByLine, kTilesByLine, kNoFilter, nullptr, 1.f,
                              nullptr, true);
  launch_columns<kColForward>(s, s.work, s.spectrum, kTilesByRow, kTilesByLine);
}

// The timer, begun by the caller, ends after pass (1): the filter's kernel.
// ftab: the smoothing's factor table, or NULL (the factors evaluated).
static void launch_inverse512(const SmootherT<float>& s, int filter, const RadialFilter& rf,
                              float norm, float* out, KernelTimer* timer, const BelowList& below,
                              const float* ftab) {
  constexpr uint32_t N = 512;
  const float* w = (s.window_mode && filter != kFilterNone) ? s.win.as<float>() : nullptr;
  if (ftab)
    launch_columns<kColTable>(s, s.spectrum, s.work, kTilesByLine, kTilesByRow, rf, w, norm, ftab);
  else
    launch_columns<kColEvaluate>(s, s.spectrum, s.work, kTilesByLine, kTilesByRow, rf, w, norm);
  if (timer) timer->end(s.stream);
  launch_columns<kColInverse>(s, s.work, s.work, kTilesByLine, kTilesByLine);
  c2r512_rows_kernel<<<N * N / kRowsPerCta, 16 * kRowsPerCta, 0, s.stream>>>(
      s.work.as<float2>(), out, (const float2*)s.twiddles, below);
  SIFG_LAUNCH_CHECK();
}
static void launch_inverse512(const SmootherT<double>&, int, const RadialFilter&, double, double*,
                              KernelTimer*, const BelowList&, const float*) {}

static int g_factor_tables = 1;
void set_factor_tables(int on) { g_factor_tables = on; }

static RadialFilter radial_filter_of(int filter, double factor, double gfactor) {
  const float f = (float)factor;
  return RadialFilter{filter == kFilterTopHat || filter == kFilterGaussian ? filter : kFilterNone,
                      (float)(factor * factor), (float)(0.5 * gfactor * gfactor), f,
                      (float)(factor - (double)f)};
}

template <class R>
const float* SmootherT<R>::factor_table(int filter, R r, R sigma) {
  if constexpr (sizeof(R) != 4) {
    return nullptr;
  } else {
    if (!g_factor_tables || !twiddles || filter == kFilterNone) return nullptr;
    factor_clock++;
    for (auto& t : factor_tables)
      if (t->filter == filter && t->r == r && t->sigma == sigma && t->box == box &&
          t->window_mode == window_mode) {
        t->used = factor_clock;
        return t->buf.template as<float>();
      }
    std::unique_ptr<FactorTable> t;
    if ((int)factor_tables.size() >= kFactorTables) {
      auto lru = std::min_element(factor_tables.begin(), factor_tables.end(),
                                  [](const auto& a, const auto& b) { return a->used < b->used; });
      t = std::move(*lru);
      factor_tables.erase(lru);
    } else {
      t.reset(new FactorTable);
    }
    t->filter = filter;
    t->r = r;
    t->sigma = sigma;
    t->box = box;
    t->window_mode = window_mode;
    t->used = factor_clock;
    float* tab = (float*)t->buf.ensure((size_t)kFactorSide * kFactorSide * kFactorSide * sizeof(float));
    const double factor = (double)r * 2.0 * M_PI / (double)box;
    const double gfactor = sigma > R(0) ? (double)sigma * 2.0 * M_PI / (double)box : 0.0;
    const float norm = (float)(1.0 / ((double)n * n * n));
    factor_table_kernel<<<152u * 8u, 256, 0, stream>>>(tab, radial_filter_of(filter, factor, gfactor),
                                                       window_mode ? win.template as<float>() : nullptr,
                                                       norm);
    SIFG_LAUNCH_CHECK();
    factor_tables.push_back(std::move(t));
    return factor_tables.back()->buf.template as<float>();
  }
}

template <class R>
void SmootherT<R>::smooth(int filter, R r, R sigma, R* out, KernelTimer* timer,
                          const BelowList* below, int lane, const R* table) {
  const double factor = (double)r * 2.0 * M_PI / (double)box;
  const double gfactor = sigma > R(0) ? (double)sigma * 2.0 * M_PI / (double)box : 0.0;
  const R norm = (R)(1.0 / ((double)n * n * n));
  if (sizeof(R) == 4 && twiddles) {
    // The own inverse reads the smoothing's factor table (built on first use)
    // or evaluates the radial factor as it applies it.
    const RadialFilter rf = radial_filter_of(filter, factor, gfactor);
    const float* ftab = factor_table(filter, r, sigma);
    if (timer) timer->begin(stream);
    launch_inverse512(*this, filter, rf, norm, out, timer, below ? *below : BelowList{}, ftab);
    return;
  }
  const cudaStream_t st = lane ? extra[lane - 1].st : stream;
  const DevBuf& lwork = lane ? extra[lane - 1].work : work;
  const cufftHandle plan = lane ? extra[lane - 1].c2r : plan_c2r;
  if (!table) table = tables(filter, &r, &sigma, 1, lane ? extra[lane - 1].lut : lut, st);
  if constexpr (sizeof(R) == 8) {
    if (twiddles) {
      const double* w = window_mode && filter != kFilterNone ? win.template as<double>() : nullptr;
      fft64_inverse(n, spectrum.template as<double2>(), lwork.as<double2>(), out, table, w, norm,
                    (const double*)twiddles, st, timer);
      return;
    }
  }
  if (timer) timer->begin(st);
  launch_filter(*this, filter, norm, table, lwork, st);
  SIFG_LAUNCH_CHECK();
  if (timer) timer->end(st);
  if (sizeof(R) == 8)
    SIFG_CUFFT(cufftExecZ2D(plan, (cufftDoubleComplex*)lwork.ptr, (cufftDoubleReal*)out));
  else
    SIFG_CUFFT(cufftExecC2R(plan, (cufftComplex*)lwork.ptr, (cufftReal*)out));
}

template <class R>
void SmootherT<R>::restore(R* out) {
  smooth(kFilterNone, R(0), R(0), out, nullptr);
}

template struct SmootherT<float>;
template struct SmootherT<double>;

}  // namespace sifg
