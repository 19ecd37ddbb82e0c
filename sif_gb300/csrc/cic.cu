// CIC deposit of particles onto the density grid, and the density contrast.
//
// Replaces grid_compute_cic / grid_cic_deposit_tile (src/structures/grid.c:
// 455-746) and sif_grid_to_density_contrast (grid.c:1177-1244).
//
// The reference sums float weights in a fixed slab/chunk order so its grid is
// deterministic. Here every corner weight is quantised to 2^-24 of a particle
// and summed as int64, so the sum is exact and independent of the order the
// GPU happens to add in. The eight quantised weights of a particle sum to
// exactly 2^24: each corner is rounded, and what rounding left over goes to
// the particle's largest corner.
//
// Layout of the work:
//   1. tile_count:   each particle's tile (16^3 base cells), histogram with
//                    warp-aggregated atomics;
//   2. exclusive scan of the tile counts;
//   3. tile_scatter: each particle's base cell and fractions, found once, as
//                    a 16-byte record in tile order (one atomic per group of
//                    lanes bound for the same tile);
//   4. tile_deposit: one CTA per tile accumulates a 17^3 tile of 64-bit sums
//                    (32-bit words plus carries) in shared memory with one
//                    shared atomic per corner; the 15^3 cells no other tile touches
//                    are written straight to the grid as float density, the
//                    faces shared with neighbouring tiles go to int64 face
//                    buffers with global atomics;
//   5. face_fixup:   the face buffers converted to float density.
//
// Weighted (sif_field_t::weights), a particle's corners carry its weight as
// the reference's products do (grid.c:635-639: the weight times each z
// factor, then the (x, y) products times those), quantised to 2^-24 of the
// binade of the largest weight magnitude: the same integers as unweighted
// when every weight is that power of two, so weights of 1 or 4 give the
// unweighted density times the weight, bit for bit. Negative weights sum as
// two's complement; a non-finite weight deposits nothing in the sums and
// its products are added to its eight cells afterwards, so those cells go
// non-finite as the reference's do.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace sifg {

constexpr int TB = kCicTile;  // base cells per tile side
constexpr int TS = TB + 1;    // tile extent including the upper neighbours

struct CicGeom {
  uint32_t n;       // grid cells per side
  uint32_t nt;      // tiles per side
  float box;
  float idx_hi;     // n / box in double, as a pair of floats
  float idx_lo;
  float margin;     // 2^-21 n: see cic_axis_inner
  float last;       // n as a float
};

// A coordinate in cell units, u = fold(v) * n / box, and its base cell and
// fraction (grid.c:585-620: cell = floor(u), wrapped into [0, n); t = u -
// floor(u)). The reference rounds u to a float, which moves t by up to an
// ulp of u -- 1e-5 of a cell at u ~ 128; here the product is kept exact as
// hi + lo (lo from the fused multiply-add's residual), so t is good to an ulp
// of 1 and the deposit's error is the 2^-24 quantum.
__device__ __forceinline__ void cic_axis(float v, const CicGeom& g, uint32_t& cell, float& t) {
  const float x = box_fold(v, g.box);
  const float hi = fmul(x, g.idx_hi);
  const float lo = fadd(__fmaf_rn(x, g.idx_hi, -hi), fmul(x, g.idx_lo));
  float r = floorf(hi);
  float f = fadd(fsub(hi, r), lo);
  if (f < 0.0f) {
    r -= 1.0f;
    f = fadd(f, 1.0f);
  } else if (f >= 1.0f) {
    r += 1.0f;
    f = fsub(f, 1.0f);
  }
  int32_t c = (int32_t)r;
  if (c < 0) c += (int32_t)g.n;
  if (c >= (int32_t)g.n) c -= (int32_t)g.n;
  // In range for every position in the box; the clamp only keeps a position
  // far outside it (which the box check reports) from indexing past the grid.
  cell = min((uint32_t)c, g.n - 1);
  t = f;
}

// The same for a position well inside its cell, without the fold, the carries
// and the clamp: v in [0, box) folds to itself, and where hi lies further from
// the integers than |lo| can reach -- lo is at most half an ulp of hi plus x *
// idx_lo, below 2^-22 n together, for hi <= n -- the floor of hi is u's and
// hi - floor(hi) + lo needs no carry. False, for the general form to decide,
// outside that: 2^-21 n of the positions (NaN among them), since every
// comparison must hold.
__device__ __forceinline__ bool cic_axis_inner(float v, const CicGeom& g, uint32_t& cell, float& t) {
  const float hi = fmul(v, g.idx_hi);
  const float lo = fadd(__fmaf_rn(v, g.idx_hi, -hi), fmul(v, g.idx_lo));
  const float r = floorf(hi);
  const float f0 = fsub(hi, r);
  cell = (uint32_t)(int32_t)r;
  t = fadd(f0, lo);
  return v >= 0.0f && v < g.box && hi < g.last && f0 > g.margin && f0 < 1.0f - g.margin;
}

// A particle's base cell (and fractions): most take the short form, and the
// two give the same bits where both apply.
__device__ __forceinline__ void cic_particle(float x, float y, float z, const CicGeom& g,
                                             uint32_t (&c)[3], float (&t)[3]) {
  const bool bx = cic_axis_inner(x, g, c[0], t[0]), by = cic_axis_inner(y, g, c[1], t[1]),
             bz = cic_axis_inner(z, g, c[2], t[2]);
  if (!(bx && by && bz)) {
    cic_axis(x, g, c[0], t[0]);
    cic_axis(y, g, c[1], t[1]);
    cic_axis(z, g, c[2], t[2]);
  }
}

__device__ __forceinline__ uint32_t tile_index(const uint32_t (&c)[3], const CicGeom& g) {
  return ((c[0] / TB) * g.nt + c[1] / TB) * g.nt + c[2] / TB;
}

// Both passes of the tile sort were bound by their instructions (a particle's
// three folds, carries and clamps), not by their traffic: the short form of
// cic_particle, and kSortUnroll particles' loads, matches and atomics in
// flight a thread.
constexpr int kSortT = 256;
constexpr int kSortUnroll = 4;

// With `outside` set, also counts the particles outside [lo, hi] on any axis
// (NaN included): the box check, from the same reads.
__global__ void __launch_bounds__(kSortT) tile_count_kernel(
    const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z, uint64_t n,
    CicGeom g, uint32_t* __restrict__ counts, float lo, float hi,
    unsigned long long* __restrict__ outside) {
  const uint64_t stride = (uint64_t)gridDim.x * kSortT * kSortUnroll;
  uint32_t bad = 0;
  for (uint64_t base = (uint64_t)blockIdx.x * kSortT * kSortUnroll; base < n; base += stride) {
    float px[kSortUnroll], py[kSortUnroll], pz[kSortUnroll];
    uint32_t tile[kSortUnroll];
#pragma unroll
    for (int u = 0; u < kSortUnroll; u++) {
      const uint64_t p = base + u * kSortT + threadIdx.x;
      if (p < n) {
        px[u] = x[p];
        py[u] = y[p];
        pz[u] = z[p];
      }
    }
#pragma unroll
    for (int u = 0; u < kSortUnroll; u++) {
      tile[u] = 0xffffffffu;
      if (base + u * kSortT + threadIdx.x < n) {
        uint32_t c[3];
        float t[3];
        cic_particle(px[u], py[u], pz[u], g, c, t);
        tile[u] = tile_index(c, g);
        const float mn = fminf(fminf(px[u], py[u]), pz[u]), mx = fmaxf(fmaxf(px[u], py[u]), pz[u]);
        // fminf and fmaxf pass over a NaN: the sum of the three keeps it.
        bad += (mn >= lo && mx <= hi && px[u] + py[u] + pz[u] == px[u] + py[u] + pz[u]) ? 0u : 1u;
      }
    }
#pragma unroll
    for (int u = 0; u < kSortUnroll; u++) {
      const unsigned peers = __match_any_sync(0xffffffffu, tile[u]);
      if (tile[u] != 0xffffffffu && (threadIdx.x & 31u) == (unsigned)(__ffs(peers) - 1))
        atomicAdd(counts + tile[u], (uint32_t)__popc(peers));
    }
  }
  if (outside) {
    unsigned long long b = __reduce_add_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31u) == 0 && b) atomicAdd(outside, b);
  }
}

// A particle's deposit record: its fractions along x, y, z and, in the
// fourth word's bits, its base cell within its tile (x << 8 | y << 4 | z).
static_assert(TB == 16, "4 bits per axis of the cell within its tile");

__global__ void __launch_bounds__(kSortT) tile_scatter_kernel(
    const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z, uint64_t n,
    CicGeom g, uint32_t* __restrict__ cursor, float4* __restrict__ rec, const float* __restrict__ w,
    float* __restrict__ wrec) {
  const uint64_t stride = (uint64_t)gridDim.x * kSortT * kSortUnroll;
  const unsigned lane = threadIdx.x & 31u;
  for (uint64_t base = (uint64_t)blockIdx.x * kSortT * kSortUnroll; base < n; base += stride) {
    float px[kSortUnroll], py[kSortUnroll], pz[kSortUnroll];
    float4 r[kSortUnroll];
    uint32_t slot[kSortUnroll], tile[kSortUnroll], peers[kSortUnroll];
#pragma unroll
    for (int u = 0; u < kSortUnroll; u++) {
      const uint64_t p = base + u * kSortT + threadIdx.x;
      if (p < n) {
        px[u] = x[p];
        py[u] = y[p];
        pz[u] = z[p];
      }
    }
#pragma unroll
    for (int u = 0; u < kSortUnroll; u++) {
      tile[u] = 0xffffffffu;
      if (base + u * kSortT + threadIdx.x < n) {
        uint32_t c[3];
        float t[3];
        cic_particle(px[u], py[u], pz[u], g, c, t);
        tile[u] = tile_index(c, g);
        r[u] = make_float4(t[0], t[1], t[2],
                           __uint_as_float((c[0] % TB) << 8 | (c[1] % TB) << 4 | (c[2] % TB)));
      }
    }
#pragma unroll
    for (int u = 0; u < kSortUnroll; u++) {
      peers[u] = __match_any_sync(0xffffffffu, tile[u]);
      if (tile[u] != 0xffffffffu && lane == (unsigned)(__ffs(peers[u]) - 1))
        slot[u] = atomicAdd(cursor + tile[u], (uint32_t)__popc(peers[u]));
    }
#pragma unroll
    for (int u = 0; u < kSortUnroll; u++) {
      const uint32_t s = __shfl_sync(0xffffffffu, slot[u], __ffs(peers[u]) - 1) +
                         __popc(peers[u] & ((1u << lane) - 1u));
      if (tile[u] != 0xffffffffu) {
        rec[s] = r[u];
        if (w) wrec[s] = w[base + u * kSortT + threadIdx.x];
      }
    }
  }
}

// The largest finite weight magnitude, as its bits (which order as the
// magnitudes do), and the count of non-finite weights.
__global__ void weight_max_kernel(const float* __restrict__ w, uint64_t n,
                                  unsigned* __restrict__ out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned m = 0, bad = 0;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    const unsigned b = __float_as_uint(w[p]) & 0x7fffffffu;
    if (b >= 0x7f800000u)
      bad++;
    else
      m = max(m, b);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  bad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31u) == 0) {
    if (m) atomicMax(out, m);
    if (bad) atomicAdd(out + 1, bad);
  }
}

// The weighted quantum from the largest weight's binade [2^E, 2^(E+1)):
// corners quantised at 2^(E-24) (scale 2^(24-E)), clamped to keep both the
// scale and its inverse normal floats.
__device__ __forceinline__ int weight_scale_exp(const unsigned* wmax) {
  const int e = (int)(*wmax >> 23) - 127;
  return min(100, max(-100, 24 - e));
}

// Each non-finite weight's eight products, added to its cells after the
// deposit (the reference's float sums carry them into those cells).
__global__ void nonfinite_weights_kernel(const float* __restrict__ x, const float* __restrict__ y,
                                         const float* __restrict__ z,
                                         const float* __restrict__ w, uint64_t n, CicGeom g,
                                         const unsigned* __restrict__ wmax,
                                         float* __restrict__ grid) {
  if (wmax[1] == 0) return;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    const float pw = w[p];
    if ((__float_as_uint(pw) & 0x7fffffffu) < 0x7f800000u) continue;
    uint32_t c[3];
    float t[3];
    cic_axis(x[p], g, c[0], t[0]);
    cic_axis(y[p], g, c[1], t[1]);
    cic_axis(z[p], g, c[2], t[2]);
    for (int k = 0; k < 8; k++) {
      uint32_t q[3];
      float f = 1.0f;
      for (int a = 0; a < 3; a++) {
        const int up = (k >> (2 - a)) & 1;
        q[a] = up ? (c[a] + 1 == g.n ? 0u : c[a] + 1) : c[a];
        f = fmul(f, up ? t[a] : fsub(1.0f, t[a]));
      }
      float* cell = grid + ((uint64_t)q[0] * g.n + q[1]) * g.n + q[2];
      *cell = fadd(*cell, fmul(pw, f));
    }
  }
}

// Face buffers: cells on a tile boundary in x (x % TB == 0), else in y, else
// in z, each laid out densely over its own boundary planes.
struct FaceBufs {
  unsigned long long* fx;  // [nt][n][n]
  unsigned long long* fy;  // [n][nt][n]
  unsigned long long* fz;  // [n][n][nt]
};

__device__ __forceinline__ unsigned long long* face_slot(const FaceBufs& f, uint32_t gx,
                                                        uint32_t gy, uint32_t gz,
                                                        const CicGeom& g) {
  const uint64_t n = g.n, nt = g.nt;
  if (gx % TB == 0) return f.fx + ((uint64_t)(gx / TB) * n + gy) * n + gz;
  if (gy % TB == 0) return f.fy + ((uint64_t)gx * nt + gy / TB) * n + gz;
  return f.fz + ((uint64_t)gx * n + gy) * nt + gz / TB;
}

// A particle's eight corner quanta (corner k at x + (k >> 2 & 1), y + (k >> 1
// & 1), z + (k & 1)), which sum to exactly `whole`: the reference's products
// (grid.c:627-650), (x, y) pairs times z (wz0, wz1: times the weight), each
// rounded, and the remainder added to the first largest.
__device__ __forceinline__ void corner_quanta(float tx, float ty, float wz0, float wz1,
                                              float qscale, int whole, uint32_t (&q)[8]) {
  const float wx0 = fsub(1.0f, tx), wy0 = fsub(1.0f, ty);
  const float w00 = fmul(wx0, wy0), w01 = fmul(wx0, ty);
  const float w10 = fmul(tx, wy0), w11 = fmul(tx, ty);
  const float w[8] = {fmul(w00, wz0), fmul(w00, wz1), fmul(w01, wz0), fmul(w01, wz1),
                      fmul(w10, wz0), fmul(w10, wz1), fmul(w11, wz0), fmul(w11, wz1)};
  // w times a power of two is exact in float, so rounding it to an
  // integer in float is the quantisation itself; GB300's FP64 rate is
  // no place for it.
  int sum = 0;
  int big = 0;
  float wbig = fabsf(w[0]);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int qk = __float2int_rn(fmul(w[k], qscale));
    q[k] = (uint32_t)qk;
    sum += qk;
    if (fabsf(w[k]) > wbig) {  // the first largest, as a scan from corner 0 finds it
      wbig = fabsf(w[k]);
      big = k;
    }
  }
  const int fix = whole - sum;
#pragma unroll
  for (int k = 0; k < 8; k++) q[k] = (uint32_t)((int)q[k] + (k == big ? fix : 0));
}

constexpr int kWhole = 16777216;  // one particle, in quanta of 2^-24
constexpr int kTileWords = TS * TS * TS;
constexpr int kDepositT = 256;

__device__ __forceinline__ uint32_t tile_cell(uint32_t local) {
  return ((local >> 8) * TS + ((local >> 4) & 15u)) * TS + (local & 15u);
}
__device__ __forceinline__ uint32_t corner_offset(int k) {
  return (uint32_t)(((k >> 2) & 1) * TS * TS + ((k >> 1) & 1) * TS + (k & 1));
}

// A tile's place in the grid: its first node and its extent.
struct TilePlace {
  uint32_t ox, oy, oz, ex, ey, ez;
  __device__ __forceinline__ TilePlace(uint32_t tile, const CicGeom& g) {
    const uint32_t nt = g.nt;
    ox = tile / (nt * nt) * TB;
    oy = (tile / nt) % nt * TB;
    oz = tile % nt * TB;
    ex = min((uint32_t)TB, g.n - ox);
    ey = min((uint32_t)TB, g.n - oy);
    ez = min((uint32_t)TB, g.n - oz);
  }
};

// One particle's corners added into a tile's words.
__device__ __forceinline__ void add_particle(const float4& r, uint32_t* acc) {
  constexpr float qscale = (float)kWhole;
  const float wx0 = fsub(1.0f, r.x), wy0 = fsub(1.0f, r.y), wz0 = fsub(1.0f, r.z);
  const float w00 = fmul(wx0, wy0), w01 = fmul(wx0, r.y);
  const float w10 = fmul(r.x, wy0), w11 = fmul(r.x, r.y);
  const float w[8] = {fmul(w00, wz0), fmul(w00, r.z), fmul(w01, wz0), fmul(w01, r.z),
                      fmul(w10, wz0), fmul(w10, r.z), fmul(w11, wz0), fmul(w11, r.z)};
  uint32_t* cell = acc + tile_cell(__float_as_uint(r.w));
  uint32_t sum = 0, big = 0;
  float wbig = w[0];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint32_t q = __float_as_uint(__fmaf_rn(w[k], qscale, 8388608.0f)) - 0x4b000000u;
    atomicAdd(cell + corner_offset(k), q);
    sum += q;
    if (k > 0 && w[k] > wbig) {  // the first largest, as corner_quanta finds it
      wbig = w[k];
      big = corner_offset(k);
    }
  }
  atomicAdd(cell + big, (uint32_t)kWhole - sum);
}

// A node of a tile, at (a, b, c) of it: straight to the grid where no other
// tile touches it, else to its face buffer; nothing where it lies past the grid.
__device__ __forceinline__ void put_node(const TilePlace& t, const CicGeom& g, uint32_t a, uint32_t b,
                                         uint32_t c, unsigned long long v, float qinv, float inv_cell_vol,
                                         float* __restrict__ grid, const FaceBufs& faces) {
  if (a > t.ex || b > t.ey || c > t.ez) return;
  const uint32_t gx = t.ox + a == g.n ? 0u : t.ox + a;
  const uint32_t gy = t.oy + b == g.n ? 0u : t.oy + b;
  const uint32_t gz = t.oz + c == g.n ? 0u : t.oz + c;
  if (a >= 1 && a < t.ex && b >= 1 && b < t.ey && c >= 1 && c < t.ez)
    grid[((uint64_t)gx * g.n + gy) * g.n + gz] =
        fmul(fmul(__ll2float_rn((long long)v), qinv), inv_cell_vol);
  else if (v != 0ull)
    atomicAdd(face_slot(faces, gx, gy, gz, g), v);
}

// The unweighted deposit, one CTA a tile at a time: the tile's sums as one
// 32-bit word a cell, one shared atomic a corner. The word's wraps are not
// watched add by add: every quantum is non-negative (the weights are, and the
// remainder of a few quanta goes to a corner of at least 2^21), so the words
// of a tile sum to its particles times 2^24 exactly when none of them wrapped,
// and each wrap takes 2^32 from that sum. A tile whose sum falls short (a cell
// of 256 particles or more) is left to tile_dense_kernel, through `redo`
// (redo[0] counts them), as is one of more than `dense` particles, which all but
// surely has such a cell.
// (Two words a cell, as the wide kernel keeps, cost a second atomic a corner:
// the 512^3 deposit 1.57 ms in 39 KB of shared memory a CTA, 1.23 with one.)
//
// The kernel is bound by its instructions. A corner's quantum is rounded by
// adding 2^23 to it (an fma; an integer conversion runs at a quarter of the
// rate): exact for every weight up to a half. The largest corner's can be
// more, and whatever its bits then say, the remainder -- what the eight lack
// of one particle, added modulo 2^32 to the same word by a ninth atomic --
// makes it the particle's rest: the same quanta as corner_quanta's, without
// a select per corner to place the remainder. The flush takes the tile's
// inside and its faces in passes of their own, each cell's place a few
// instructions (one loop over all 17^3 with a test of each cell's kind was
// half of the kernel).
__global__ void __launch_bounds__(kDepositT, 6) tile_deposit_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ offsets, CicGeom g,
    float inv_cell_vol, float* __restrict__ grid, FaceBufs faces, uint32_t dense,
    uint32_t* __restrict__ redo) {
  __shared__ uint32_t acc[kTileWords];
  __shared__ unsigned long long wsum[kDepositT / 32];
  const uint32_t n_tiles = g.nt * g.nt * g.nt;
  constexpr float qinv = 1.0f / (float)kWhole;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  // Cleared once; each flush leaves the cells it reads cleared for the next tile.
  for (int i = threadIdx.x; i < kTileWords; i += kDepositT) acc[i] = 0u;
  __syncthreads();
  for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const uint32_t s = offsets[tile], e = offsets[tile + 1];
    if (e - s > dense) {
      if (threadIdx.x == 0) redo[1 + atomicAdd(redo, 1u)] = tile;
      continue;
    }
    for (uint32_t p = s + threadIdx.x; p < e; p += kDepositT) add_particle(__ldg(rec + p), acc);
    __syncthreads();
    unsigned long long sum = 0;
    for (int i = threadIdx.x; i < kTileWords; i += kDepositT) sum += acc[i];
    // A lane's sum is below 20 * 2^32: in two parts whose warp sums fit.
    const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)sum & 0xfffffu);
    const uint32_t hi = __reduce_add_sync(0xffffffffu, (uint32_t)(sum >> 20));
    if (lane == 0) wsum[warp] = ((unsigned long long)hi << 20) + lo;
    __syncthreads();
    sum = 0;
#pragma unroll
    for (int w = 0; w < kDepositT / 32; w++) sum += wsum[w];
    if (sum != (unsigned long long)(e - s) << 24) {
      if (threadIdx.x == 0) redo[1 + atomicAdd(redo, 1u)] = tile;
      for (int i = threadIdx.x; i < kTileWords; i += kDepositT) acc[i] = 0u;
      __syncthreads();
      continue;
    }

    // The flush: nodes 1 .. e-1 of the tile on every axis are touched by no
    // other tile and go straight to the grid, a half-warp a z row; the rest to
    // the face buffers, each in face_slot's order of precedence. Cells past
    // the grid's end hold nothing.
    const TilePlace t(tile, g);
    const uint32_t n = g.n;
    for (uint32_t row = threadIdx.x >> 4; row < (TB - 1) * (TB - 1); row += kDepositT / 16) {
      const uint32_t a = 1 + row / (TB - 1), b = 1 + row % (TB - 1), c = 1 + (threadIdx.x & 15u);
      if (a < t.ex && b < t.ey && c < t.ez) {
        uint32_t* src = acc + (a * TS + b) * TS + c;
        grid[(size_t)((t.ox + a) * n + t.oy + b) * n + t.oz + c] =
            fmul(fmul(__uint2float_rn(*src), qinv), inv_cell_vol);
        *src = 0u;
      }
    }
    auto to_face = [&](uint32_t a, uint32_t b, uint32_t c, unsigned long long* slot) {
      uint32_t* src = acc + (a * TS + b) * TS + c;
      const uint32_t v = *src;
      *src = 0u;
      if (v) atomicAdd(slot, (unsigned long long)v);
    };
    auto wrap = [&](uint32_t v) { return v == n ? 0u : v; };
    for (uint32_t i = threadIdx.x; i < 2 * TS * TS; i += kDepositT) {
      const uint32_t a = i < TS * TS ? 0u : t.ex, b = i / TS % TS, c = i % TS;
      if (b <= t.ey && c <= t.ez)
        to_face(a, b, c,
                faces.fx + ((size_t)(wrap(t.ox + a) / TB) * n + wrap(t.oy + b)) * n + wrap(t.oz + c));
    }
    for (uint32_t i = threadIdx.x; i < 2 * (TB - 1) * TS; i += kDepositT) {
      const uint32_t b = i < (TB - 1) * TS ? 0u : t.ey, a = 1 + i / TS % (TB - 1), c = i % TS;
      if (a < t.ex && c <= t.ez)
        to_face(a, b, c,
                faces.fy + ((size_t)(t.ox + a) * g.nt + wrap(t.oy + b) / TB) * n + wrap(t.oz + c));
    }
    for (uint32_t i = threadIdx.x; i < 2 * (TB - 1) * (TB - 1); i += kDepositT) {
      const uint32_t c = i < (TB - 1) * (TB - 1) ? 0u : t.ez, a = 1 + i / (TB - 1) % (TB - 1),
                     b = 1 + i % (TB - 1);
      if (a < t.ex && b < t.ey)
        to_face(a, b, c,
                faces.fz + (size_t)((t.ox + a) * n + t.oy + b) * g.nt + wrap(t.oz + c) / TB);
    }
    __syncthreads();
  }
}

// The tiles with a cell of 256 particles or more, listed by the kernel above:
// each cell's sum from two passes over the tile's particles in the one word a
// cell, the quanta modulo 2^32 and then the quanta over 2^12. A word of up to
// kDensePart particles' quanta over 2^12 does not wrap, and times 2^12 falls
// short of their sum by less than 2^12 a particle: the sum is the one number
// within 2^32 from there up with those low 32 bits. A tile of more particles
// takes that many at a time. Most tiles of a clustered snapshot come here, and
// the kernel ends with its densest: kDenseUnroll records in flight a thread, and
// two CTAs an SM, which a thread's twenty sums in registers leave room for (half
// of 16.7 M particles in haloes, on 256^3: 1.193 ms a deposit with one, 1.158
// with two, 1.231 with three, spilling).
//
// (Two words a cell in one pass over the particles, one CTA an SM as so few
// were expected: half of 16.7 M particles in haloes, on 200^3, 2.37 ms a
// deposit, now 1.61; every tile that way from the first, 1.98. In the kernel
// above, which has the first pass's words: 0.110 to 0.117 ms for 16.7 M uniform
// particles' tiles, none of them dense.)
constexpr uint32_t kDensePart = (1u << 20) - 1;
constexpr int kDenseUnroll = 4;
template <class Each>
__device__ __forceinline__ void each_record(const float4* __restrict__ rec, uint32_t s, uint32_t e, Each each) {
  for (uint32_t p = s + threadIdx.x; p < e; p += kDenseUnroll * kDepositT) {
    float4 r[kDenseUnroll];
#pragma unroll
    for (int u = 0; u < kDenseUnroll; u++)
      if (p + u * kDepositT < e) r[u] = __ldg(rec + p + u * kDepositT);
#pragma unroll
    for (int u = 0; u < kDenseUnroll; u++)
      if (p + u * kDepositT < e) each(r[u]);
  }
}

__global__ void __launch_bounds__(kDepositT, 2) tile_dense_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ offsets, CicGeom g,
    float inv_cell_vol, float* __restrict__ grid, FaceBufs faces, const uint32_t* __restrict__ redo) {
  __shared__ uint32_t acc[kTileWords];
  constexpr int kPer = (kTileWords + kDepositT - 1) / kDepositT;  // words a thread
  const uint32_t n_items = redo[0];
  if (blockIdx.x >= n_items) return;
  for (int i = threadIdx.x; i < kTileWords; i += kDepositT) acc[i] = 0u;
  __syncthreads();
  for (uint32_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    const uint32_t tile = redo[1 + item], s = offsets[tile], e = offsets[tile + 1];
    unsigned long long v[kPer] = {};
    for (uint32_t p0 = s, p1; p0 < e; p0 = p1) {
      p1 = p0 + min(kDensePart, e - p0);
      each_record(rec, p0, p1, [&](const float4& r) { add_particle(r, acc); });
      __syncthreads();
      uint32_t lo[kPer];
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const uint32_t i = threadIdx.x + j * kDepositT;
        if (i >= kTileWords) break;
        lo[j] = acc[i];
        acc[i] = 0u;
      }
      __syncthreads();
      each_record(rec, p0, p1, [&](const float4& r) {
        uint32_t q[8];
        corner_quanta(r.x, r.y, fsub(1.0f, r.z), r.z, (float)kWhole, kWhole, q);
        uint32_t* cell = acc + tile_cell(__float_as_uint(r.w));
#pragma unroll
        for (int k = 0; k < 8; k++) atomicAdd(cell + corner_offset(k), q[k] >> 12);
      });
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const uint32_t i = threadIdx.x + j * kDepositT;
        if (i >= kTileWords) break;
        const unsigned long long least = (unsigned long long)acc[i] << 12;
        v[j] += least + (uint32_t)(lo[j] - (uint32_t)least);
        acc[i] = 0u;
      }
      __syncthreads();
    }
    const TilePlace t(tile, g);
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const uint32_t i = threadIdx.x + j * kDepositT;
      if (i >= kTileWords) break;
      put_node(t, g, i / (TS * TS), i / TS % TS, i % TS, v[j], 1.0f / (float)kWhole, inv_cell_vol, grid,
               faces);
    }
  }
}

// The weighted deposit. Two 32-bit words a cell: a 32-bit shared atomic add is
// one instruction, a 64-bit one a compare-and-swap loop
// (measured: the 512^3 deposit with one 64-bit add per corner took 3.4 ms,
// against 1.7). A tile with fewer than 2^16 particles adds each quantum's low
// 16 bits to the first word and its high bits (arithmetic shift) to the
// second, neither of which can wrap (a cell takes one add per particle), with
// adds that return nothing; a denser tile adds the whole quantum to the first
// word and counts its wraps in the second (each add is below 2^32, so it wraps
// at most once), which needs the old value back. Either pair is the exact
// 64-bit sum whatever the order of the adds.
__global__ void __launch_bounds__(kDepositT) tile_deposit_wide_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ offsets, CicGeom g,
    float inv_cell_vol, float* __restrict__ grid, FaceBufs faces,
    const float* __restrict__ wrec, const unsigned* __restrict__ wmax) {
  extern __shared__ uint32_t acc_lo[];  // TS^3 words, then TS^3 carries
  uint32_t* acc_hi = acc_lo + kTileWords;
  const uint32_t n_tiles = g.nt * g.nt * g.nt;
  // The quantum: 2^-24 of the largest weight's binade.
  const int we = weight_scale_exp(wmax);
  const float qscale = __uint_as_float((uint32_t)(127 + we) << 23);
  const float qinv = __uint_as_float((uint32_t)(127 - we) << 23);
  // Cleared once; each flush leaves the cells it reads cleared for the next tile.
  for (int i = threadIdx.x; i < 2 * kTileWords; i += kDepositT) acc_lo[i] = 0u;
  __syncthreads();
  for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const uint32_t s = offsets[tile], e = offsets[tile + 1];
    const bool split = e - s < (1u << 16);
    for (uint32_t p = s + threadIdx.x; p < e; p += kDepositT) {
      const float4 r = __ldg(rec + p);
      // A non-finite weight is added afterwards, outside the sums.
      float pw = __ldg(wrec + p);
      if ((__float_as_uint(pw) & 0x7fffffffu) >= 0x7f800000u) pw = 0.0f;
      uint32_t q[8];
      corner_quanta(r.x, r.y, fmul(pw, fsub(1.0f, r.z)), fmul(pw, r.z), qscale,
                    __float2int_rn(fmul(pw, qscale)), q);  // summing to the weight's own quanta
      const uint32_t cell = tile_cell(__float_as_uint(r.w));
      // One shared atomic per word and corner. (Reducing lanes bound for the
      // same cell first with __reduce_add_sync over each lane group's own mask
      // costs a serialised pass per distinct group: eight per corner per cell
      // in the warp, far more than the atomics it saves.)
      if (split) {
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint32_t c = cell + corner_offset(k);
          atomicAdd(acc_lo + c, q[k] & 0xffffu);
          const int hi16 = (int)q[k] >> 16;
          if (hi16) atomicAdd(acc_hi + c, (uint32_t)hi16);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint32_t v = q[k];
          const uint32_t c = cell + corner_offset(k);
          const uint32_t old = atomicAdd(acc_lo + c, v);
          // The carry, and for a negative value its sign extension.
          const uint32_t hi = (old + v < old ? 1u : 0u) + ((int)v < 0 ? 0xffffffffu : 0u);
          if (hi) atomicAdd(acc_hi + c, hi);
        }
      }
    }
    __syncthreads();
    const TilePlace t(tile, g);
    for (int i = threadIdx.x; i < kTileWords; i += kDepositT) {
      const unsigned long long v =
          split ? (unsigned long long)((long long)(int)acc_hi[i] * 65536ll + (long long)acc_lo[i])
                : ((unsigned long long)acc_hi[i] << 32) | acc_lo[i];
      acc_lo[i] = 0u;
      acc_hi[i] = 0u;
      put_node(t, g, i / (TS * TS), i / TS % TS, i % TS, v, qinv, inv_cell_vol, grid, faces);
    }
    __syncthreads();
  }
}

// The face buffers converted to density: blockIdx.y is a buffer and one of
// its nt shares of n^2 entries (in x and y, a boundary plane). A plane past the
// grid's end holds nothing, and a node on an earlier buffer's planes belongs
// to that buffer.
__global__ void face_fixup_kernel(CicGeom g, float inv_cell_vol, float* __restrict__ grid,
                                  FaceBufs faces, const unsigned* __restrict__ wmax) {
  float qinv = 1.0f / 16777216.0f;
  if (wmax) qinv = __uint_as_float((uint32_t)(127 - weight_scale_exp(wmax)) << 23);
  const uint32_t n = g.n, nt = g.nt;
  const uint32_t which = blockIdx.y / nt, k = blockIdx.y % nt;
  if (which < 2 && k * TB >= n) return;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n * n; j += gridDim.x * blockDim.x) {
    const uint32_t u = j / n, v = j % n;
    uint32_t gx, gy, gz;
    const unsigned long long* from;
    if (which == 0) {
      gx = k * TB, gy = u, gz = v;
      from = faces.fx + (size_t)k * n * n + j;
    } else if (which == 1) {
      gx = u, gy = k * TB, gz = v;
      if (gx % TB == 0) continue;
      from = faces.fy + ((size_t)gx * nt + k) * n + gz;
    } else {
      // The buffer's z planes lie next to one another: its k-th n^2 entries.
      const size_t i = (size_t)k * n * n + j;
      const size_t line = i < 0xffffffffull ? (uint32_t)i / nt : i / nt;
      gx = (uint32_t)line / n, gy = (uint32_t)line % n, gz = (uint32_t)(i - line * nt) * TB;
      if (gx % TB == 0 || gy % TB == 0 || gz >= n) continue;
      from = faces.fz + i;
    }
    grid[(size_t)(gx * n + gy) * n + gz] =
        fmul(fmul(__ll2float_rn((long long)*from), qinv), inv_cell_vol);
  }
}

// ---------------------------------------------------------------------------
// The FP64 form's deposit (the reference's SIF_USE_DOUBLE build): the cell
// coordinate u = fold(x) * (N / L), its base cell and fraction, and the eight
// weights in double as grid.c:585-650 computes them. Each weight is rounded to
// a multiple of 2^-40 of a particle (the remainder to the largest, so the
// eight sum to exactly one particle) and summed as int64 with global atomics:
// the grid is exact to 2^-40 per particle and independent of the order the
// additions land in. One thread per particle, no tiling: this is the plain
// form the float path is measured against.
//
// The FP64 pipe (two lanes a clock an SM) bounded it before the atomics did: of
// the sixty FP64 instructions a particle took, the box's comparisons, the
// conversions to and from whole numbers and the choice of the largest weight go
// by integers, and a weight is rounded to its quantum by one addition. 16.7 M
// particles on 256^3: 2.06 to 1.21 ms.
// ---------------------------------------------------------------------------
constexpr double kQ64 = 1099511627776.0;  // 2^40

__device__ __forceinline__ void cic_axis_f64(double v, uint32_t n, double box, double idx,
                                             uint32_t& c0, uint32_t& c1, double& t) {
  uint32_t raw;
  if (in_box(v, box)) {
    // The whole part by integers, as a double by clearing the bits below it.
    const double u = fmul(v, idx);
    raw = whole_part(u);
    const uint32_t hi = (uint32_t)__double2hiint(u) & 0x7fffffffu, lo = (uint32_t)__double2loint(u);
    const int e = (int)(hi >> 20) - 1023;
    const double w = e < 0    ? 0.0
                     : e < 20 ? __hiloint2double((int)(hi & (0xffffffffu << (20 - e))), 0)
                              : __hiloint2double((int)hi, e == 20 ? 0 : (int)(lo & (0xffffffffu << (52 - e))));
    t = fsub(u, w);
  } else {
    const double u = fmul(box_fold(v, box), idx);
    raw = (uint32_t)u;
    t = fsub(u, (double)raw);
  }
  c0 = raw >= n ? 0u : raw;
  c1 = c0 + 1 == n ? 0u : c0 + 1;
}

// Weighted: the largest finite weight magnitude's bits and the count of
// non-finite weights, as weight_max_kernel in float.
__global__ void weight_max_f64_kernel(const double* __restrict__ w, uint64_t n,
                                      unsigned long long* __restrict__ out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long m = 0, bad = 0;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(w[p]) & 0x7fffffffffffffffull;
    if (b >= 0x7ff0000000000000ull)
      bad++;
    else
      m = b > m ? b : m;
  }
  for (int d = 16; d > 0; d >>= 1) {
    const unsigned long long o = __shfl_down_sync(0xffffffffu, m, d);
    m = o > m ? o : m;
    bad += __shfl_down_sync(0xffffffffu, bad, d);
  }
  if ((threadIdx.x & 31u) == 0) {
    if (m) atomicMax(out, m);
    if (bad) atomicAdd(out + 1, bad);
  }
}

// The FP64 quantum: 2^-40 of a particle, or of the largest weight's binade
// (clamped to keep the scale and its inverse normal).
__device__ __forceinline__ int weight_scale_exp_f64(const unsigned long long* wmax) {
  const int e = (int)(wmax[0] >> 52) - 1023;
  return min(900, max(-900, 40 - e));
}

template <bool kWeighted>
__global__ void cic_f64_kernel(const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, uint64_t np, uint32_t n, double box,
                               double idx, unsigned long long* __restrict__ acc,
                               const double* __restrict__ wts,
                               const unsigned long long* __restrict__ wmax) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  double qs = kQ64;
  if (kWeighted) qs = __longlong_as_double((long long)(1023 + weight_scale_exp_f64(wmax)) << 52);
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np; p += stride) {
    uint32_t x0, x1, y0, y1, z0, z1;
    double tx, ty, tz;
    cic_axis_f64(x[p], n, box, idx, x0, x1, tx);
    cic_axis_f64(y[p], n, box, idx, y0, y1, ty);
    cic_axis_f64(z[p], n, box, idx, z0, z1, tz);
    double wz0 = fsub(1.0, tz), wz1 = tz, pw = 1.0;
    if (kWeighted) {
      pw = wts[p];
      // A non-finite weight is added afterwards, outside the sums.
      if (((unsigned long long)__double_as_longlong(pw) & 0x7fffffffffffffffull) >=
          0x7ff0000000000000ull)
        continue;
      wz0 = fmul(pw, wz0);
      wz1 = fmul(pw, wz1);
    }
    const double wx0 = fsub(1.0, tx), wy0 = fsub(1.0, ty);
    const double w00 = fmul(wx0, wy0), w01 = fmul(wx0, ty), w10 = fmul(tx, wy0),
                 w11 = fmul(tx, ty);
    const double w[8] = {fmul(w00, wz0), fmul(w00, wz1), fmul(w01, wz0), fmul(w01, wz1),
                         fmul(w10, wz0), fmul(w10, wz1), fmul(w11, wz0), fmul(w11, wz1)};
    long long q[8];
    long long sum = 0;
    int big = 0;
    auto bits = [](double v) { return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull; };
#pragma unroll
    for (int k = 0; k < 8; k++) {
      // Rounded to the quantum, to nearest even. A product of at most 1 added
      // to 1.5 2^12, whose last place is 2^-40, is rounded there by that one
      // addition, the quanta left in its low bits.
      constexpr double kPlace = 6144.0;
      if (kWeighted)
        q[k] = __double2ll_rn(fmul(w[k], qs));
      else
        q[k] = __double_as_longlong(__dadd_rn(w[k], kPlace)) - 0x40b8000000000000ll;  // kPlace's bits
      sum += q[k];
      if (bits(w[k]) > bits(w[big])) big = k;
    }
    const long long fix = (kWeighted ? __double2ll_rn(fmul(pw, qs)) : (long long)kQ64) - sum;
    const uint32_t xs[2] = {x0, x1}, ys[2] = {y0, y1}, zs[2] = {z0, z1};
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const long long v = q[k] + (k == big ? fix : 0);
      if (v == 0) continue;
      const uint64_t c = ((uint64_t)xs[k >> 2] * n + ys[(k >> 1) & 1]) * n + zs[k & 1];
      atomicAdd(acc + c, (unsigned long long)v);
    }
  }
}

__global__ void cic_f64_finish_kernel(const unsigned long long* __restrict__ acc, uint64_t cells,
                                      double inv_cell_vol, double* __restrict__ grid,
                                      const unsigned long long* __restrict__ wmax) {
  double qinv = 1.0 / kQ64;
  if (wmax) qinv = __longlong_as_double((long long)(1023 - weight_scale_exp_f64(wmax)) << 52);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cells; i += stride)
    grid[i] = fmul(fmul(__ll2double_rn((long long)acc[i]), qinv), inv_cell_vol);
}

// Each non-finite weight's eight products added to its cells (see the float
// form's nonfinite_weights_kernel).
__global__ void nonfinite_weights_f64_kernel(const double* __restrict__ x,
                                             const double* __restrict__ y,
                                             const double* __restrict__ z,
                                             const double* __restrict__ w, uint64_t np, uint32_t n,
                                             double box, double idx,
                                             const unsigned long long* __restrict__ wmax,
                                             double* __restrict__ grid) {
  if (wmax[1] == 0) return;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np; p += stride) {
    const double pw = w[p];
    if (((unsigned long long)__double_as_longlong(pw) & 0x7fffffffffffffffull) <
        0x7ff0000000000000ull)
      continue;
    uint32_t c0[3], c1[3];
    double t[3];
    cic_axis_f64(x[p], n, box, idx, c0[0], c1[0], t[0]);
    cic_axis_f64(y[p], n, box, idx, c0[1], c1[1], t[1]);
    cic_axis_f64(z[p], n, box, idx, c0[2], c1[2], t[2]);
    for (int k = 0; k < 8; k++) {
      uint32_t q[3];
      double f = 1.0;
      for (int a = 0; a < 3; a++) {
        const int up = (k >> (2 - a)) & 1;
        q[a] = up ? c1[a] : c0[a];
        f = fmul(f, up ? t[a] : fsub(1.0, t[a]));
      }
      double* cell = grid + ((uint64_t)q[0] * n + q[1]) * n + q[2];
      *cell = fadd(*cell, fmul(pw, f));
    }
  }
}

size_t cic_f64_scratch_bytes(uint32_t n) { return (size_t)n * n * n * sizeof(unsigned long long) + 512; }

void cic_deposit_f64(const double* x, const double* y, const double* z, uint64_t n_particles,
                     uint32_t n, double box, double* grid, void* scratch, cudaStream_t st,
                     KernelTimer* timer, const double* w) {
  const uint64_t cells = (uint64_t)n * n * n;
  unsigned long long* acc = (unsigned long long*)scratch;
  unsigned long long* wmax = w ? acc + cells : nullptr;
  SIFG_CUDA(cudaMemsetAsync(acc, 0, (cells + (w ? 2 : 0)) * sizeof(unsigned long long), st));
  // grid.c:684 and 735-737 in double.
  const double idx = (double)n / box;
  const double cl = box / (double)n;
  const double inv_cell_vol = 1.0f / (double)(cl * cl * cl);
  if (w) {
    weight_max_f64_kernel<<<grid_for(n_particles, 256, 152u * 16u), 256, 0, st>>>(w, n_particles,
                                                                                  wmax);
    SIFG_LAUNCH_CHECK();
  }
  if (timer) timer->begin(st);
  (w ? cic_f64_kernel<true> : cic_f64_kernel<false>)<<<grid_for(n_particles, 256), 256, 0, st>>>(
      x, y, z, n_particles, n, box, idx, acc, w, wmax);
  SIFG_LAUNCH_CHECK();
  if (timer) timer->end(st);
  cic_f64_finish_kernel<<<grid_for(cells, 256), 256, 0, st>>>(acc, cells, inv_cell_vol, grid, wmax);
  SIFG_LAUNCH_CHECK();
  if (w) {
    nonfinite_weights_f64_kernel<<<grid_for(n_particles, 256, 152u * 16u), 256, 0, st>>>(
        x, y, z, w, n_particles, n, box, idx, wmax, grid);
    SIFG_LAUNCH_CHECK();
  }
}

// ---------------------------------------------------------------------------
// Density contrast: the mean in double over fixed blocks (a fixed launch, so
// the summation order and the result never change), then v * inv - 1.
// ---------------------------------------------------------------------------
constexpr int kMeanBlocks = 1024;
constexpr int kMeanThreads = 256;

template <class R>
__global__ void __launch_bounds__(kMeanThreads) mean_partial_kernel(const R* __restrict__ v,
                                                                    uint64_t n,
                                                                    double* __restrict__ partial) {
  __shared__ double s[kMeanThreads];
  const uint64_t chunk = (n + kMeanBlocks - 1) / kMeanBlocks;
  const uint64_t lo = (uint64_t)blockIdx.x * chunk;
  const uint64_t hi = lo + chunk < n ? lo + chunk : n;
  double acc = 0.0;
  // Four loads in flight, added in the same order as one at a time.
  uint64_t i = lo + threadIdx.x;
  for (; i + 3 * kMeanThreads < hi; i += 4 * kMeanThreads) {
    const R a = v[i], b = v[i + kMeanThreads], c = v[i + 2 * kMeanThreads],
            d = v[i + 3 * kMeanThreads];
    acc += (double)a;
    acc += (double)b;
    acc += (double)c;
    acc += (double)d;
  }
  for (; i < hi; i += kMeanThreads) acc += (double)v[i];
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int w = kMeanThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// The float form's partial sums without a double operation per value: this
// GPU's FP64 rate would bound the pass (a conversion and an add per cell),
// not its 4 bytes a cell. Each thread keeps its running sum as a float pair
// by Knuth's TwoSum (the rounding error of every add kept in the low part),
// at least as exact as a double chain over the same values, in the same
// fixed order; the block's 256 pairs are then added in double as above.
template <>
__global__ void __launch_bounds__(kMeanThreads) mean_partial_kernel<float>(
    const float* __restrict__ v, uint64_t n, double* __restrict__ partial) {
  __shared__ double s[kMeanThreads];
  const uint64_t chunk = (n + kMeanBlocks - 1) / kMeanBlocks;
  const uint64_t lo = (uint64_t)blockIdx.x * chunk;
  const uint64_t hi = lo + chunk < n ? lo + chunk : n;
  float sh = 0.0f, sl = 0.0f;
  auto add = [&](float x) {
    const float t = __fadd_rn(sh, x);
    const float b = __fsub_rn(t, sh);
    const float e = __fadd_rn(__fsub_rn(sh, __fsub_rn(t, b)), __fsub_rn(x, b));
    sh = t;
    sl = __fadd_rn(sl, e);
  };
  uint64_t i = lo + threadIdx.x;
  for (; i + 3 * kMeanThreads < hi; i += 4 * kMeanThreads) {
    const float a = v[i], b = v[i + kMeanThreads], c = v[i + 2 * kMeanThreads],
                d = v[i + 3 * kMeanThreads];
    add(a);
    add(b);
    add(c);
    add(d);
  }
  for (; i < hi; i += kMeanThreads) add(v[i]);
  s[threadIdx.x] = (double)sh + (double)sl;
  __syncthreads();
  for (int w = kMeanThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// The blocks' sums added by pairs, in a fixed order: eleven dependent adds
// and one load deep. (One thread adding 1,024 of them in a row took 56 us.)
__global__ void __launch_bounds__(kMeanBlocks / 2) mean_final_kernel(
    const double* __restrict__ partial, uint64_t n, double* __restrict__ mean_out) {
  __shared__ double s[kMeanBlocks / 2];
  s[threadIdx.x] = partial[threadIdx.x] + partial[threadIdx.x + kMeanBlocks / 2];
  __syncthreads();
  for (int w = kMeanBlocks / 4; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) mean_out[0] = s[0] / (double)n;
}

// Sixteen bytes a load and store (v is 16-byte aligned), the values past the
// last whole ones by the last block's first threads. From the end backwards:
// the mean's pass, just before it, left the end of the grid in L2.
template <class R>
__global__ void __launch_bounds__(256) contrast_kernel(R* __restrict__ v, uint64_t n,
                                                       const double* __restrict__ mean) {
  // The double division once a block (this GPU's FP64 rate is low).
  __shared__ R inv_s;
  if (threadIdx.x == 0) inv_s = (R)(1.0 / mean[0]);
  __syncthreads();
  const R inv = inv_s;
  constexpr uint32_t kPer = 16 / sizeof(R);
  struct alignas(16) Pack {
    R v[kPer];
  };
  Pack* packs = (Pack*)v;
  const uint64_t np = n / kPer, stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < np; i += 2 * stride) {
    const bool two = i + stride < np;
    Pack a = packs[np - 1 - i], b{};
    if (two) b = packs[np - 1 - i - stride];
#pragma unroll
    for (uint32_t k = 0; k < kPer; k++) {
      a.v[k] = fsub(fmul(a.v[k], inv), R(1.0f));
      b.v[k] = fsub(fmul(b.v[k], inv), R(1.0f));
    }
    packs[np - 1 - i] = a;
    if (two) packs[np - 1 - i - stride] = b;
  }
  const uint64_t i = np * kPer + threadIdx.x;
  if (blockIdx.x == gridDim.x - 1 && i < n) v[i] = fsub(fmul(v[i], inv), R(1.0f));
}

// The same, one value a thread, where v is not 16-byte aligned.
template <class R>
__global__ void contrast_any_kernel(R* __restrict__ v, uint64_t n, const double* __restrict__ mean) {
  __shared__ R inv_s;
  if (threadIdx.x == 0) inv_s = (R)(1.0 / mean[0]);
  __syncthreads();
  const R inv = inv_s;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    v[i] = fsub(fmul(v[i], inv), R(1.0f));
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

static CicGeom make_geom(uint32_t n, float box) {
  CicGeom g;
  g.n = n;
  g.nt = (n + TB - 1) / TB;
  g.box = box;
  const double idx = (double)n / (double)box;
  g.idx_hi = (float)idx;
  g.idx_lo = (float)(idx - (double)g.idx_hi);
  g.margin = (float)n / 2097152.0f;
  g.last = (float)n;
  return g;
}

size_t cic_scratch_bytes(uint64_t n_particles, uint32_t n, bool weighted) {
  const uint64_t nt = (n + TB - 1) / TB;
  const uint64_t tiles = nt * nt * nt;
  const uint64_t face = 3 * nt * (uint64_t)n * n * sizeof(unsigned long long);
  return n_particles * (sizeof(float4) + (weighted ? sizeof(float) : 0)) +
         (2 * tiles + 2) * sizeof(uint32_t) + face + 16 * 256 + 512;
}

// The deposit's scratch, laid out.
struct CicScratch {
  float4* rec;
  uint32_t *counts, *cursor;
  FaceBufs faces;
  float* wrec;
  unsigned* wmax;
  size_t face_elems;
  uint64_t tiles;
  CicScratch(void* scratch, uint64_t n_particles, uint32_t n, const CicGeom& g, bool weighted) {
    char* p = (char*)scratch;
    auto take = [&](size_t bytes) {
      char* r = p;
      p += (bytes + 255) & ~(size_t)255;
      return (void*)r;
    };
    tiles = (uint64_t)g.nt * g.nt * g.nt;
    face_elems = (size_t)g.nt * n * n;
    rec = (float4*)take(n_particles * sizeof(float4));
    counts = (uint32_t*)take((tiles + 1) * sizeof(uint32_t));
    cursor = (uint32_t*)take((tiles + 1) * sizeof(uint32_t));
    faces.fx = (unsigned long long*)take(face_elems * 8);
    faces.fy = (unsigned long long*)take(face_elems * 8);
    faces.fz = (unsigned long long*)take(face_elems * 8);
    wrec = weighted ? (float*)take(n_particles * sizeof(float)) : nullptr;
    wmax = weighted ? (unsigned*)take(2 * sizeof(unsigned)) : nullptr;
  }
};

static void tile_count(const float* x, const float* y, const float* z, uint64_t n_particles,
                       const CicGeom& g, const CicScratch& b, cudaStream_t st, const float* bounds,
                       unsigned long long* outside) {
  SIFG_CUDA(cudaMemsetAsync(b.counts, 0, (b.tiles + 1) * sizeof(uint32_t), st));
  tile_count_kernel<<<grid_for(n_particles, kSortT * kSortUnroll, 152u * 8u), kSortT, 0, st>>>(
      x, y, z, n_particles, g, b.counts, bounds ? bounds[0] : 0.f, bounds ? bounds[1] : 0.f,
      bounds ? outside : nullptr);
  SIFG_LAUNCH_CHECK();
}

void cic_count(const float* x, const float* y, const float* z, uint64_t n_particles, uint32_t n,
               float box, void* scratch, cudaStream_t st, const float* bounds,
               unsigned long long* outside) {
  const CicGeom g = make_geom(n, box);
  SIFG_CUDA(cudaMemsetAsync(outside, 0, sizeof(*outside), st));
  // The weights' buffers lie after everything this pass touches.
  tile_count(x, y, z, n_particles, g, CicScratch(scratch, n_particles, n, g, false), st, bounds, outside);
}

void cic_deposit(const float* x, const float* y, const float* z, uint64_t n_particles,
                 uint32_t n, float box, float* grid, void* scratch, cudaStream_t st,
                 KernelTimer* timer, const float* bounds, unsigned long long* outside,
                 cudaEvent_t sorted, const float* w, KernelTimer* stage, bool counted) {
  const CicGeom g = make_geom(n, box);
  const CicScratch b(scratch, n_particles, n, g, w != nullptr);

  // The stage: the tile sort, the deposit proper and the faces' fix-up.
  if (stage) stage->begin(st);
  SIFG_CUDA(cudaMemsetAsync(b.faces.fx, 0, (char*)(b.faces.fz + b.face_elems) - (char*)b.faces.fx, st));
  if (w) {
    SIFG_CUDA(cudaMemsetAsync(b.wmax, 0, 2 * sizeof(unsigned), st));
    weight_max_kernel<<<grid_for(n_particles, 256, 152u * 16u), 256, 0, st>>>(w, n_particles, b.wmax);
    SIFG_LAUNCH_CHECK();
  }
  if (!counted) tile_count(x, y, z, n_particles, g, b, st, bounds, outside);
  exclusive_scan_u32(b.counts, (uint32_t)(b.tiles + 1), st);
  SIFG_CUDA(cudaMemcpyAsync(b.cursor, b.counts, (b.tiles + 1) * sizeof(uint32_t),
                            cudaMemcpyDeviceToDevice, st));
  tile_scatter_kernel<<<grid_for(n_particles, kSortT * kSortUnroll, 152u * 8u), kSortT, 0, st>>>(
      x, y, z, n_particles, g, b.cursor, b.rec, w, b.wrec);
  SIFG_LAUNCH_CHECK();
  if (sorted) SIFG_CUDA(cudaEventRecord(sorted, st));
  const float cl = box / (float)n;
  const float inv_cell_vol = 1.0f / (float)(cl * cl * cl);
  const size_t smem = (size_t)2 * kTileWords * sizeof(uint32_t);
  auto grid_of = [&](unsigned per_sm) { return (unsigned)std::min<uint64_t>(b.tiles, 152u * per_sm); };
  if (timer) timer->begin(st);
  if (w) {
    tile_deposit_wide_kernel<<<grid_of(5), kDepositT, smem, st>>>(b.rec, b.counts, g, inv_cell_vol, grid,
                                                                  b.faces, b.wrec, b.wmax);
    SIFG_LAUNCH_CHECK();
  } else {
    // The scatter's cursors are free: the list of tiles to do again. A tile of
    // eight particles a node and four times the box's mean is taken for one of
    // them unseen: it would be found to be one after a pass of its own (haloes
    // on 200^3 1.93 ms, 1.60 with the rule).
    uint32_t* redo = b.cursor;
    const uint64_t dense = std::min<uint64_t>(
        std::max<uint64_t>(4 * n_particles / b.tiles, 8u * TB * TB * TB), kDensePart);
    SIFG_CUDA(cudaMemsetAsync(redo, 0, sizeof(uint32_t), st));
    tile_deposit_kernel<<<grid_of(6), kDepositT, 0, st>>>(b.rec, b.counts, g, inv_cell_vol, grid, b.faces,
                                                          (uint32_t)dense, redo);
    SIFG_LAUNCH_CHECK();
    tile_dense_kernel<<<grid_of(4), kDepositT, 0, st>>>(b.rec, b.counts, g, inv_cell_vol, grid, b.faces,
                                                        redo);
    SIFG_LAUNCH_CHECK();
  }
  if (timer) timer->end(st);
  face_fixup_kernel<<<dim3(grid_for((uint64_t)n * n, 256, 152u * 16u), 3 * g.nt), 256, 0, st>>>(
      g, inv_cell_vol, grid, b.faces, b.wmax);
  SIFG_LAUNCH_CHECK();
  if (stage) stage->end(st);
  if (w) {
    nonfinite_weights_kernel<<<grid_for(n_particles, 256, 152u * 16u), 256, 0, st>>>(
        x, y, z, w, n_particles, g, b.wmax, grid);
    SIFG_LAUNCH_CHECK();
  }
}

template <class R>
void density_contrast(R* v, uint64_t n, double* d_scratch, cudaStream_t st, bool mean_only) {
  // d_scratch: kMeanBlocks + 1 doubles.
  mean_partial_kernel<R><<<kMeanBlocks, kMeanThreads, 0, st>>>(v, n, d_scratch);
  SIFG_LAUNCH_CHECK();
  mean_final_kernel<<<1, kMeanBlocks / 2, 0, st>>>(d_scratch, n, d_scratch + kMeanBlocks);
  SIFG_LAUNCH_CHECK();
  if (!mean_only) apply_contrast(v, n, d_scratch + kMeanBlocks, st);
}
template void density_contrast<float>(float*, uint64_t, double*, cudaStream_t, bool);
template void density_contrast<double>(double*, uint64_t, double*, cudaStream_t, bool);

template <class R>
void apply_contrast(R* v, uint64_t n, const double* mean, cudaStream_t st) {
  if ((uintptr_t)v % 16 == 0)
    contrast_kernel<R><<<grid_for(n * sizeof(R) / 32, 256, 152u * 8u), 256, 0, st>>>(v, n, mean);
  else
    contrast_any_kernel<R><<<grid_for(n, 256), 256, 0, st>>>(v, n, mean);
  SIFG_LAUNCH_CHECK();
}
template void apply_contrast<float>(float*, uint64_t, const double*, cudaStream_t);
template void apply_contrast<double>(double*, uint64_t, const double*, cudaStream_t);

const double* contrast_mean(const double* d_scratch) { return d_scratch + kMeanBlocks; }

size_t density_contrast_scratch_bytes() { return (kMeanBlocks + 1) * sizeof(double); }

double read_mean(const double* d_scratch, cudaStream_t st) {
  // On the stream that computed it: the library's streams do not wait for
  // the legacy default stream, nor it for them.
  double m = 0.0;
  SIFG_CUDA(cudaMemcpyAsync(&m, d_scratch + kMeanBlocks, sizeof(double), cudaMemcpyDeviceToHost, st));
  SIFG_CUDA(cudaStreamSynchronize(st));
  return m;
}

}  // namespace sifg
