// The FP64 form's transforms on cubic grids of 128 and 256 cells a side:
// the forward R2C and, per smoothing, the filter and the inverse C2R, three
// passes each (kx, ky as columns of the half spectrum, kz as rows).
//
// What bounds them is the FP64 pipe: two fused multiply-adds a clock an SM,
// 630 G/s for the GPU, against some 40 us of memory traffic a pass at 256^3.
// A pass takes its count of FP64 instructions over that rate and everything
// else -- the shared memory exchanges, the integer work of quarter turns, the
// filter's gathers -- runs beside it. So the transforms are laid out to need
// few of them, and every one that can be is a fused multiply-add:
//
//   A rotation by an angle of at most pi/4 is cos (1 + i tan): the two fused
//   multiply-adds of (1 + i tan) are applied and the cos is carried as the
//   element's scale (as Linzer and Feig, 1993, and Goedecker, 1997, lay out
//   transforms for fused multiply-adds). A butterfly of two elements of scales a and b takes
//   x +- (b / a) y, four fused multiply-adds as four additions would have
//   been, and leaves scale a. Quarter turns, which bring every angle within
//   pi/4, are exchanges of parts and signs and no arithmetic. Decimation in
//   frequency turns element 0 of every block by nothing, so the scale left at
//   the end is 1. The ratios are constants of the code within a transform and
//   come from a table where a twiddle between two stages is taken in.
//
// A 16-point transform is 148 instructions, 178 with its twiddles; a
// 256-point column 5,216 (a fused radix-16 with whole complex products:
// 6,200), a row of 256 reals 2,900. 256^3, at the pipe's rate and measured: the
// pass that filters 315 and 350 us, the other columns 274 and 317, the rows 300
// and 361; cuFFT's three passes and the filter kernel took 1,870 a smoothing
// (here 1,030). Against the identity the error is 4.8e-16 rms, 5.6e-16 before.
//
// 64^3 stays with cuFFT: CTAs of this size leave three quarters of the SMs
// without one (203 us a forward and inverse, 156 there); 128^3 356 and 577.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "common.cuh"
#include "smooth.cuh"

namespace sifg {
namespace {

constexpr int kThreads = 256;
constexpr int kPoints = 16;  // values a thread holds
constexpr int kSlots = kThreads * kPoints;

// ---------------------------------------------------------------------------
// The transform of P <= 16 points in registers, e^{+2 pi i jk / P}
// ---------------------------------------------------------------------------
constexpr double kTan8 = 0.41421356237309504880;  // tan(pi/8)
// |cos| of e pi / 8 brought within pi/4 by quarter turns.
__host__ __device__ constexpr double turn_scale(int e) {
  return e % 4 == 0 ? 1.0 : e % 4 == 2 ? 0.70710678118654752440 : 0.92387953251128675613;
}
// The scale of element i before level `level` (blocks of P >> level), from
// the turns of the levels above.
__host__ __device__ constexpr double level_scale(int P, int level, int i) {
  if (level == 0) return 1.0;
  const int p = P >> (level - 1), h = p / 2, off = i % p;
  return off < h ? level_scale(P, level - 1, i)
                 : level_scale(P, level - 1, i - h) * turn_scale((off - h) * 16 / p);
}
// The ratio b / a of butterfly `k` (of P / 2) of a level.
__host__ __device__ constexpr double level_ratio(int P, int level, int k) {
  const int p = P >> level, h = p / 2, a = k / h * p + k % h;
  return level_scale(P, level, a + h) / level_scale(P, level, a);
}
__host__ __device__ constexpr int levels(int P) { return P == 1 ? 0 : 1 + levels(P / 2); }
// Where the transform leaves output k: the bits of k turned round.
__host__ __device__ constexpr int turned(int P, int k) {
  int r = 0;
  for (int b = 1; b < P; b <<= 1) r = 2 * r + ((k & b) ? 1 : 0);
  return r;
}

// d turned by e pi / 8, its scale turn_scale(e) left out.
template <int E>
__device__ __forceinline__ double2 turn(double2 d) {
  constexpr double t = kTan8;
  if constexpr (E == 0) return d;
  if constexpr (E == 1) return make_double2(fma(-t, d.y, d.x), fma(t, d.x, d.y));
  if constexpr (E == 2) return make_double2(d.x - d.y, d.x + d.y);
  if constexpr (E == 3) return make_double2(fma(t, d.x, -d.y), fma(t, d.y, d.x));
  if constexpr (E == 4) return make_double2(-d.y, d.x);
  if constexpr (E == 5) return make_double2(fma(-t, d.x, -d.y), fma(-t, d.y, d.x));
  if constexpr (E == 6) return make_double2(-d.x - d.y, d.x - d.y);
  return make_double2(fma(-t, d.y, -d.x), fma(t, d.x, -d.y));
}

template <int P, int L, int I, bool kTw>
__device__ __forceinline__ void butterfly(double2 (&v)[P], const double* __restrict__ ratio) {
  constexpr int p = P >> L, h = p / 2, a = I / h * p + I % h, e = I % h * 16 / p;
  constexpr double k = level_ratio(P, L, I);
  const double2 x = v[a], y = v[a + h];
  double2 s, d;
  if constexpr (!kTw && k == 1.0) {
    s = make_double2(x.x + y.x, x.y + y.y);
    d = make_double2(x.x - y.x, x.y - y.y);
  } else {
    const double r = kTw ? __ldg(ratio + (L * (P / 2) + I) * 16) : k;
    s = make_double2(fma(r, y.x, x.x), fma(r, y.y, x.y));
    d = make_double2(fma(-r, y.x, x.x), fma(-r, y.y, x.y));
  }
  v[a] = s;
  v[a + h] = turn<e>(d);
}
template <int P, int L, bool kTw, int... I>
__device__ __forceinline__ void level_of(double2 (&v)[P], const double* __restrict__ ratio,
                                         std::integer_sequence<int, I...>) {
  (butterfly<P, L, I, kTw>(v, ratio), ...);
}
template <int P, bool kTw, int... L>
__device__ __forceinline__ void all_levels(double2 (&v)[P], const double* __restrict__ ratio,
                                           std::integer_sequence<int, L...>) {
  (level_of<P, L, kTw>(v, ratio, std::make_integer_sequence<int, P / 2>{}), ...);
}
// Output k in v[turned(P, k)]. With kTw the elements come with the scales
// the table's ratios are made for (twiddle()).
template <int P, bool kTw>
__device__ __forceinline__ void dft(double2 (&v)[P], const double* __restrict__ ratio = nullptr) {
  all_levels<P, kTw>(v, ratio, std::make_integer_sequence<int, levels(P)>{});
}

// x times i^q, without the FP64 pipe.
__device__ __forceinline__ double2 quarter_turns(double2 x, uint32_t q) {
  const int xh = __double2hiint(x.x), xl = __double2loint(x.x);
  const int yh = __double2hiint(x.y), yl = __double2loint(x.y);
  const int flip = (int)((q & 2u) << 30);
  const bool odd = q & 1u;
  return make_double2(
      __hiloint2double((odd ? (int)(yh ^ 0x80000000) : xh) ^ flip, odd ? yl : xl),
      __hiloint2double((odd ? xh : yh) ^ flip, odd ? xl : yl));
}

// The twiddles of a second stage: T elements of transform k1 (of 16), element
// m turned by m k1 of M parts of the circle. Laid out entry by entry, k1
// fastest: tan of each of the T - 1, the T / 2 ratios of each level, and the
// quarter turns, two bits an element, in a word.
__host__ __device__ constexpr int stage_doubles(int T) { return (T - 1 + levels(T) * (T / 2)) * 16; }

template <int T>
__device__ __forceinline__ void twiddle(double2 (&w)[T], const double* __restrict__ tab, uint32_t q) {
#pragma unroll
  for (int m = 1; m < T; m++) {
    const double t = __ldg(tab + (m - 1) * 16);
    const double2 x = quarter_turns(w[m], q >> (2 * m) & 3u);
    w[m] = make_double2(fma(-t, x.y, x.x), fma(t, x.x, x.y));
  }
}

// One device block of tables per grid size:
//   the column stage (T = N / 16), the row stage (T = N / 32), then tan and
//   cos of 2 pi k / N, k <= N / 8, of the rows' packing, and the quarter turns
//   of the two stages (16 words each).
template <int N>
struct Tables {
  static constexpr int kCol = 0;
  static constexpr int kRow = kCol + stage_doubles(N / 16);
  static constexpr int kTan = kRow + stage_doubles(N / 32);
  static constexpr int kCos = kTan + N / 8 + 1;
  static constexpr int kTurns = kCos + N / 8 + 1;
  static constexpr int kDoubles = kTurns + 16;  // 32 words
};

// ---------------------------------------------------------------------------
// kx and ky: columns
// ---------------------------------------------------------------------------
// The half spectrum is [kx][ky][kz], kz <= N / 2. Column q starts at
// (q / inner) * outer + q % inner, its elements `elem` apart: the columns of a
// pass, of whichever axis, are numbered through, so that N / 2 + 1 of them a
// line leave no CTA part empty. N / 16 threads a column, 4096 / N columns a
// CTA, neighbouring lanes on neighbouring columns.
struct Columns {
  uint32_t inner, outer, elem;
};

// The filter of the first inverse pass: mode (kx, ky, kz) by lut[|k|^2], the
// window's factor of each axis (win, or NULL) and norm, found once for +-kx.
struct Filter64 {
  const double* lut;
  const double* win;
  double norm;
};

enum Pass { kFilterPass, kInversePass, kForwardPass };

template <int N, Pass kPass>
__global__ void __launch_bounds__(kThreads, 2)
    columns64_kernel(const double2* src, double2* dst, Columns cl, const double* __restrict__ tab,
                     Filter64 f) {
  constexpr int T = N / 16, kCols = kThreads / T, kModes = N / 2 + 1;
  extern __shared__ __align__(16) double2 ex[];  // kSlots, then the filter's factors
  const uint32_t c = threadIdx.x % kCols, j = threadIdx.x / kCols;
  const uint32_t q = blockIdx.x * kCols + c;
  const size_t base = (size_t)(q / cl.inner) * cl.outer + q % cl.inner;
  double2 v[kPoints];
#pragma unroll
  for (int r = 0; r < kPoints; r++) v[r] = src[base + (size_t)(j + T * r) * cl.elem];
  if constexpr (kPass == kFilterPass) {
    double* fac = (double*)(ex + kSlots);  // by |kx|, kCols each
    double* wx = fac + kModes * kCols;
    for (uint32_t k = threadIdx.x; k < kModes; k += kThreads)
      wx[k] = f.win ? f.norm * __ldg(f.win + k) : f.norm;
    __syncthreads();
    const uint32_t ky = q / kModes, kz = q % kModes, a = ky > N / 2 ? N - ky : ky;
    const uint32_t k2 = a * a + kz * kz;
    const double wyz = f.win ? __ldg(f.win + ky) * __ldg(f.win + kz) : 1.0;
    for (uint32_t kx = j; kx < kModes; kx += T)
      fac[kx * kCols + c] = __ldg(f.lut + kx * kx + k2) * (wx[kx] * wyz);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPoints; r++) {
      const uint32_t kx = j + T * r;
      const double s = fac[(kx > N / 2 ? N - kx : kx) * kCols + c];
      v[r] = make_double2(v[r].x * s, v[r].y * s);
    }
  }
  // The forward as the conjugate of the inverse of the conjugate.
  if constexpr (kPass == kForwardPass) {
#pragma unroll
    for (int r = 0; r < kPoints; r++) v[r].y = -v[r].y;
  }
  dft<16, false>(v);
#pragma unroll
  for (int k1 = 0; k1 < 16; k1++) ex[(k1 * T + j) * kCols + c] = v[turned(16, k1)];
  __syncthreads();
  const uint32_t* turns = (const uint32_t*)(tab + Tables<N>::kTurns);
#pragma unroll
  for (int u = 0; u < 16 / T; u++) {
    const uint32_t k1 = j + T * u;
    double2 w[T];
#pragma unroll
    for (int m = 0; m < T; m++) w[m] = ex[(k1 * T + m) * kCols + c];
    const double* t = tab + Tables<N>::kCol + k1;
    twiddle<T>(w, t, __ldg(turns + k1));
    dft<T, true>(w, t + (T - 1) * 16);
#pragma unroll
    for (int k2 = 0; k2 < T; k2++) {
      double2 o = w[turned(T, k2)];
      if constexpr (kPass == kForwardPass) o.y = -o.y;
      dst[base + (size_t)(k1 + 16 * k2) * cl.elem] = o;
    }
  }
}

// ---------------------------------------------------------------------------
// kz: rows
// ---------------------------------------------------------------------------
// A row of N reals is a complex transform of M = N / 2 points, N / 32 threads
// a row. Its N / 2 + 1 modes, then its M points, stay in the row's slots of
// shared memory; the exchange between the stages turns the slots of each
// 16-point output so that neither side meets a bank twice.
template <int N>
struct Rows {
  static constexpr int M = N / 2, T = N / 32, kRows = kThreads / T, kSlot = M + 1;
  static constexpr size_t kBytes = (size_t)kRows * kSlot * sizeof(double2);
};

// The M-point transform of the row in shared memory, in place.
template <int N, bool kForward>
__device__ __forceinline__ void row_transform(double2* row, uint32_t j, const double* __restrict__ tab) {
  constexpr int T = Rows<N>::T;
  double2 v[kPoints];
#pragma unroll
  for (int r = 0; r < kPoints; r++) {
    v[r] = row[j + T * r];
    if (kForward) v[r].y = -v[r].y;
  }
  dft<16, false>(v);
  __syncwarp();
#pragma unroll
  for (int k1 = 0; k1 < 16; k1++) row[k1 * T + ((j + k1) & (T - 1))] = v[turned(16, k1)];
  __syncwarp();
  const uint32_t* turns = (const uint32_t*)(tab + Tables<N>::kTurns) + 16;
  double2 w[16 / T][T];
#pragma unroll
  for (int u = 0; u < 16 / T; u++) {
    const uint32_t k1 = j + T * u;
#pragma unroll
    for (int m = 0; m < T; m++) w[u][m] = row[k1 * T + ((m + k1) & (T - 1))];
  }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < 16 / T; u++) {
    const uint32_t k1 = j + T * u;
    const double* t = tab + Tables<N>::kRow + k1;
    twiddle<T>(w[u], t, __ldg(turns + k1));
    dft<T, true>(w[u], t + (T - 1) * 16);
#pragma unroll
    for (int k2 = 0; k2 < T; k2++) {
      double2 o = w[u][turned(T, k2)];
      if (kForward) o.y = -o.y;
      row[k1 + 16 * k2] = o;
    }
  }
  __syncwarp();
}

// The inverse: Z[0 .. M] (the imaginary parts of the ends taken as zero, as a
// C2R does) to c[k] = Fe + i Fo, Fe = Z[k] + conj Z[M-k], Fo = (Z[k] - conj
// Z[M-k]) e^{2 pi i k / N}, k and M - k together, whose inverse transform y
// gives x[2m] = Re y[m], x[2m+1] = Im y[m].
template <int N>
__global__ void __launch_bounds__(kThreads, 2)
    rows64_inverse_kernel(const double2* __restrict__ src, double* __restrict__ out,
                          const double* __restrict__ tab) {
  using RW = Rows<N>;
  constexpr int M = RW::M, T = RW::T;
  extern __shared__ __align__(16) double2 buf[];
  const double2* p = src + (size_t)blockIdx.x * (RW::kRows * RW::kSlot);
#pragma unroll 8
  for (uint32_t f = threadIdx.x; f < RW::kRows * RW::kSlot; f += kThreads) buf[f] = __ldg(p + f);
  __syncthreads();
  const uint32_t j = threadIdx.x % T;
  double2* row = buf + threadIdx.x / T * RW::kSlot;
#pragma unroll
  for (int r = 0; r <= 8; r++) {
    const uint32_t k = j + T * r;  // <= M / 2 = 8 T
    if (r == 8 && j != 0) break;
    double2 a = row[k], b = row[M - k];
    if (r == 0 && j == 0) a.y = b.y = 0.0;
    const double2 s = make_double2(a.x + b.x, a.y - b.y), d = make_double2(a.x - b.x, a.y + b.y);
    if (r < 4) {  // the angle is below pi/4: d (1 + i tan), by i cos
      const double t = __ldg(tab + Tables<N>::kTan + k), cs = __ldg(tab + Tables<N>::kCos + k);
      const double2 u = make_double2(fma(-t, d.y, d.x), fma(t, d.x, d.y));
      row[M - k] = make_double2(fma(cs, u.y, s.x), fma(cs, u.x, -s.y));
      row[k] = make_double2(fma(-cs, u.y, s.x), fma(cs, u.x, s.y));
    } else {      // a quarter turn less an angle within pi/4
      const double t = __ldg(tab + Tables<N>::kTan + M / 2 - k), cs = __ldg(tab + Tables<N>::kCos + M / 2 - k);
      const double2 u = make_double2(fma(t, d.y, d.x), fma(-t, d.x, d.y));
      row[M - k] = make_double2(fma(cs, u.x, s.x), fma(-cs, u.y, -s.y));
      row[k] = make_double2(fma(-cs, u.x, s.x), fma(-cs, u.y, s.y));
    }
  }
  __syncwarp();
  row_transform<N, false>(row, j, tab);
  __syncthreads();
  // By doubles: the caller's grid need not lie on 16 bytes.
  double* dst = out + (size_t)blockIdx.x * (RW::kRows * N);
  const double* from = (const double*)buf;
#pragma unroll 8
  for (uint32_t f = threadIdx.x; f < RW::kRows * N; f += kThreads)
    dst[f] = from[f / N * (2 * RW::kSlot) + f % N];
}

// The forward: with mean set the rows are the density and its contrast is
// taken as the contrast kernel takes it; X[k] = E + e^{-2 pi i k / N} O, E =
// (C[k] + conj C[M-k]) / 2, O = (C[k] - conj C[M-k]) / 2i, k and M - k together.
template <int N>
__global__ void __launch_bounds__(kThreads, 2)
    rows64_forward_kernel(const double* __restrict__ grid, double2* __restrict__ dst,
                          const double* __restrict__ tab, const double* __restrict__ mean) {
  using RW = Rows<N>;
  constexpr int M = RW::M, T = RW::T;
  extern __shared__ __align__(16) double2 buf[];
  __shared__ double inv_s;
  if (threadIdx.x == 0) inv_s = mean ? 1.0 / __ldg(mean) : 0.0;
  __syncthreads();
  const double inv = inv_s;
  const double* src = grid + (size_t)blockIdx.x * (RW::kRows * N);
  double* to = (double*)buf;
#pragma unroll 8
  for (uint32_t f = threadIdx.x; f < RW::kRows * N; f += kThreads) {
    double v = __ldg(src + f);
    if (mean) v = __dsub_rn(__dmul_rn(v, inv), 1.0);
    to[f / N * (2 * RW::kSlot) + f % N] = v;
  }
  __syncthreads();
  const uint32_t j = threadIdx.x % T;
  double2* row = buf + threadIdx.x / T * RW::kSlot;
  row_transform<N, true>(row, j, tab);
#pragma unroll
  for (int r = 0; r <= 8; r++) {
    const uint32_t k = j + T * r;
    if (r == 8 && j != 0) break;
    const double2 a = row[k], b = row[k == 0 ? 0 : M - k];
    const double2 s = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    const double2 d = make_double2(a.x - b.x, a.y + b.y);
    if (r < 4) {
      const double t = __ldg(tab + Tables<N>::kTan + k), cs = 0.5 * __ldg(tab + Tables<N>::kCos + k);
      const double2 u = make_double2(fma(t, d.y, d.x), fma(-t, d.x, d.y));
      row[M - k] = make_double2(fma(-cs, u.y, s.x), fma(-cs, u.x, -s.y));
      row[k] = make_double2(fma(cs, u.y, s.x), fma(-cs, u.x, s.y));
    } else {
      const double t = __ldg(tab + Tables<N>::kTan + M / 2 - k),
                   cs = 0.5 * __ldg(tab + Tables<N>::kCos + M / 2 - k);
      const double2 u = make_double2(fma(-t, d.y, d.x), fma(t, d.x, d.y));
      row[M - k] = make_double2(fma(cs, u.x, s.x), fma(-cs, u.y, -s.y));
      row[k] = make_double2(fma(-cs, u.x, s.x), fma(-cs, u.y, s.y));
    }
  }
  __syncthreads();
  double2* p = dst + (size_t)blockIdx.x * (RW::kRows * RW::kSlot);
#pragma unroll 8
  for (uint32_t f = threadIdx.x; f < RW::kRows * RW::kSlot; f += kThreads) p[f] = buf[f];
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
// 2 pi r / n as quarter turns and an angle within pi/4.
struct Angle {
  uint32_t turns;
  double tan, cos;
};
Angle angle_of(long r, long n) {
  r %= n;
  const long q = (8 * r + n) / (2 * n);  // the nearest quarter turn
  const double a = 2.0 * M_PI * (double)(4 * r - q * n) / (4.0 * (double)n);
  return {(uint32_t)(q & 3), std::tan(a), std::cos(a)};
}

// A second stage of T elements: transform k1's element m turned by m k1 of n.
void fill_stage(double* d, uint32_t* turns, int T, int n) {
  for (int k1 = 0; k1 < 16; k1++) {
    double c[16];
    uint32_t q = 0;
    for (int m = 0; m < T; m++) {
      const Angle a = angle_of((long)m * k1, n);
      c[m] = a.cos;
      q |= a.turns << (2 * m);
      if (m) d[(m - 1) * 16 + k1] = a.tan;
    }
    turns[k1] = q;
    // Element i's scale before a level: its own element's c (that of the
    // pair's lower element carried on) and the turns'.
    double* ratio = d + (T - 1) * 16;
    for (int l = 0; l < levels(T); l++)
      for (int k = 0; k < T / 2; k++) {
        const int p = T >> l, h = p / 2, m = k % h;
        ratio[(l * (T / 2) + k) * 16 + k1] = c[m + h] / c[m] * level_ratio(T, l, k);
      }
  }
}

template <int N>
std::vector<double> make_tables() {
  using TB = Tables<N>;
  std::vector<double> t(TB::kDoubles, 0.0);
  uint32_t* turns = (uint32_t*)(t.data() + TB::kTurns);
  fill_stage(t.data() + TB::kCol, turns, N / 16, N);
  fill_stage(t.data() + TB::kRow, turns + 16, N / 32, N / 2);
  for (int k = 0; k <= N / 8; k++) {
    const double a = 2.0 * M_PI * k / N;
    t[TB::kTan + k] = k == N / 8 ? 1.0 : std::tan(a);
    t[TB::kCos + k] = std::cos(a);
  }
  return t;
}

template <int N>
constexpr size_t column_bytes(bool filter) {
  constexpr int kCols = kThreads / (N / 16), kModes = N / 2 + 1;
  return kSlots * sizeof(double2) + (filter ? (size_t)kModes * (kCols + 1) * sizeof(double) : 0);
}

template <int N>
void set_smem() {
  thread_local bool attr = false;  // set once a thread: one device a process
  if (attr) return;
  SIFG_CUDA(cudaFuncSetAttribute(columns64_kernel<N, kFilterPass>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)column_bytes<N>(true)));
  SIFG_CUDA(cudaFuncSetAttribute(columns64_kernel<N, kInversePass>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)column_bytes<N>(false)));
  SIFG_CUDA(cudaFuncSetAttribute(columns64_kernel<N, kForwardPass>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)column_bytes<N>(false)));
  SIFG_CUDA(cudaFuncSetAttribute(rows64_inverse_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Rows<N>::kBytes));
  SIFG_CUDA(cudaFuncSetAttribute(rows64_forward_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Rows<N>::kBytes));
  attr = true;
}

template <int N>
struct Passes {
  static constexpr uint32_t zd = N / 2 + 1, plane = N * zd;
  static constexpr Columns kx{plane, 0, plane}, ky{zd, plane, zd};
  static constexpr unsigned kColCtas = plane * (N / 16) / kThreads, kRowCtas = N * N / Rows<N>::kRows;
  static_assert(plane * (N / 16) % kThreads == 0 && N * N % Rows<N>::kRows == 0, "whole CTAs");

  static void forward(const double* grid, const double* mean, double2* spec, const double* tab,
                      cudaStream_t st) {
    set_smem<N>();
    rows64_forward_kernel<N><<<kRowCtas, kThreads, Rows<N>::kBytes, st>>>(grid, spec, tab, mean);
    SIFG_LAUNCH_CHECK();
    for (const Columns& c : {ky, kx}) {
      columns64_kernel<N, kForwardPass>
          <<<kColCtas, kThreads, column_bytes<N>(false), st>>>(spec, spec, c, tab, Filter64{});
      SIFG_LAUNCH_CHECK();
    }
  }
  static void inverse(const double2* spec, double2* work, double* out, const double* lut,
                      const double* win, double norm, const double* tab, cudaStream_t st,
                      KernelTimer* timer) {
    set_smem<N>();
    if (timer) timer->begin(st);
    columns64_kernel<N, kFilterPass><<<kColCtas, kThreads, column_bytes<N>(true), st>>>(
        spec, work, kx, tab, Filter64{lut, win, norm});
    SIFG_LAUNCH_CHECK();
    if (timer) timer->end(st);
    columns64_kernel<N, kInversePass>
        <<<kColCtas, kThreads, column_bytes<N>(false), st>>>(work, work, ky, tab, Filter64{});
    SIFG_LAUNCH_CHECK();
    rows64_inverse_kernel<N><<<kRowCtas, kThreads, Rows<N>::kBytes, st>>>(work, out, tab);
    SIFG_LAUNCH_CHECK();
  }
};

}  // namespace

bool fft64_takes(uint32_t n) { return n == 128 || n == 256; }

std::vector<double> fft64_tables(uint32_t n) {
  return n == 128 ? make_tables<128>() : make_tables<256>();
}

void fft64_forward(uint32_t n, const double* grid, const double* mean, double2* spec,
                   const double* tab, cudaStream_t st) {
  (n == 128 ? Passes<128>::forward : Passes<256>::forward)(grid, mean, spec, tab, st);
}

void fft64_inverse(uint32_t n, const double2* spec, double2* work, double* out, const double* lut,
                   const double* win, double norm, const double* tab, cudaStream_t st,
                   KernelTimer* timer) {
  (n == 128 ? Passes<128>::inverse
            : Passes<256>::inverse)(spec, work, out, lut, win, norm, tab, st, timer);
}

}  // namespace sifg
