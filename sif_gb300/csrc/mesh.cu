// Chain-mesh build: the particles grouped by mesh cell, cells in flat order,
// each cell's particles in source order.
//
// Replaces chain_mesh_create + chain_mesh_canonicalise
// (src/structures/chain_mesh.c:680-832, 420-542). The cell of a particle is
// the reference's: (int32)(fold(x) * (1/cell_length)) clamped into the mesh
// (chain_mesh.c:316-331), so the mesh is the reference's bit for bit.
//
//   1. cell_count:  per-cell counts, warp-aggregated atomics, in scratch;
//   2. exclusive scan, copied to the cell offsets;
//   3. cell_scatter: (source index, x, y, z) into each cell's range, in the
//      order the atomics hand out slots;
//   4. cell_canon:  per entry, its rank among its cell's source indices, and
//      the entry written to that rank -- the canonical order, which no atomic
//      race can change. The rank by a warp's sort of the cell's keys (up to
//      1,024 of them; neighbouring cells of a few entries together) or, in a
//      larger cell, by a CTA's count of the smaller ones.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace sifg {

template <class R>
struct MeshGeom {
  uint32_t n;
  R box;
  R inv_l;  // 1 / cell_length
};

// A scatter record: source index and folded position.
template <class R>
struct alignas(16) MeshRec {
  uint32_t i;
  R x, y, z;
};
static_assert(sizeof(MeshRec<float>) == 16, "float records are 16 bytes");
static_assert(sizeof(MeshRec<double>) == 32, "double records are 32 bytes");

// A particle's cell, its coordinates folded into the box on the way. Nearly
// every coordinate is in [0, box), where the fold and the clamp at zero do
// nothing; any that is not (NaN among them) takes all three through them. The
// clamp into the mesh holds for what an infinite 1 / cell_length makes of a
// coordinate too (a box below about n / FLT_MAX a side).
template <class R>
__device__ __forceinline__ uint32_t mesh_cell(R& x, R& y, R& z, const MeshGeom<R>& g) {
  const uint32_t hi = g.n - 1;
  uint32_t ix, iy, iz;
  if (in_box(x, g.box) && in_box(y, g.box) && in_box(z, g.box)) {
    ix = whole_part(fmul(x, g.inv_l));
    iy = whole_part(fmul(y, g.inv_l));
    iz = whole_part(fmul(z, g.inv_l));
  } else {
    x = box_fold(x, g.box);
    y = box_fold(y, g.box);
    z = box_fold(z, g.box);
    ix = (uint32_t)max((int32_t)fmul(x, g.inv_l), 0);
    iy = (uint32_t)max((int32_t)fmul(y, g.inv_l), 0);
    iz = (uint32_t)max((int32_t)fmul(z, g.inv_l), 0);
  }
  return (min(ix, hi) * g.n + min(iy, hi)) * g.n + min(iz, hi);
}

// The passes over the particles wait on their loads and on the atomics that
// hand out slots: kMeshUnroll particles a thread in flight, U in the kernels.
// (One at a time, the scatter of 64.5 M particles into 117^3 cells spent 87% of
// its stalls on them.) One a thread up to kMeshFew particles, which do not fill
// the SMs: four in a row are the longer way there. A mesh of 10,000 particles
// 21.0 to 18.9 us past its count, of 120,000 26.1 to 24.8, of 250,000 the same.
constexpr int kMeshT = 256;
constexpr int kMeshUnroll = 4;
constexpr uint64_t kMeshFew = 1u << 17;

// With `outside` set, also counts the particles outside [lo, hi] on any axis
// (NaN included): the box check, from the same reads.
template <class R, int U>
__global__ void __launch_bounds__(kMeshT) cell_count_kernel(
    const R* __restrict__ x, const R* __restrict__ y, const R* __restrict__ z, uint64_t n,
    MeshGeom<R> g, uint32_t* __restrict__ counts, R lo, R hi,
    unsigned long long* __restrict__ outside) {
  const uint64_t stride = (uint64_t)gridDim.x * kMeshT * U;
  uint32_t bad = 0;
  for (uint64_t base = (uint64_t)blockIdx.x * kMeshT * U; base < n; base += stride) {
    R px[U], py[U], pz[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t p = base + u * kMeshT + threadIdx.x;
      if (p < n) {
        px[u] = x[p];
        py[u] = y[p];
        pz[u] = z[p];
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      uint32_t c = 0xffffffffu;
      if (base + u * kMeshT + threadIdx.x < n) {
        if (outside)
          bad += within(px[u], lo, hi) && within(py[u], lo, hi) && within(pz[u], lo, hi) ? 0u : 1u;
        c = mesh_cell(px[u], py[u], pz[u], g);
      }
      const unsigned peers = __match_any_sync(0xffffffffu, c);
      if (c != 0xffffffffu && (threadIdx.x & 31u) == (unsigned)(__ffs(peers) - 1))
        atomicAdd(counts + c, (uint32_t)__popc(peers));
    }
  }
  if (outside) {
    const unsigned long long b = __reduce_add_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31u) == 0 && b) atomicAdd(outside, b);
  }
}

// Where a scatter leaves a particle: a record with its source index, for the
// canonical order; a 16-byte position record (the float form of a build that
// leaves each cell in scatter order); the mesh's position arrays (its FP64
// form).
template <class R>
struct ToRecord {
  MeshRec<R>* tmp;
  __device__ __forceinline__ void put(uint32_t slot, uint64_t p, R x, R y, R z) const {
    MeshRec<R> rec;
    rec.i = (uint32_t)p;
    rec.x = x;
    rec.y = y;
    rec.z = z;
    tmp[slot] = rec;
  }
};
struct ToXyzw {
  float4* out;
  __device__ __forceinline__ void put(uint32_t slot, uint64_t, float x, float y, float z) const {
    out[slot] = make_float4(x, y, z, 0.f);
  }
};
template <class R>
struct ToArrays {
  R *ox, *oy, *oz;
  __device__ __forceinline__ void put(uint32_t slot, uint64_t, R x, R y, R z) const {
    ox[slot] = x;
    oy[slot] = y;
    oz[slot] = z;
  }
};

template <class R, int U, class To>
__global__ void __launch_bounds__(kMeshT) cell_scatter_kernel(
    const R* __restrict__ x, const R* __restrict__ y, const R* __restrict__ z, uint64_t n,
    MeshGeom<R> g, uint32_t* __restrict__ cursor, To to) {
  const uint64_t stride = (uint64_t)gridDim.x * kMeshT * U;
  const unsigned lane = threadIdx.x & 31u;
  for (uint64_t base = (uint64_t)blockIdx.x * kMeshT * U; base < n; base += stride) {
    R px[U], py[U], pz[U];
    uint32_t slot[U], peers[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t p = base + u * kMeshT + threadIdx.x;
      if (p < n) {
        px[u] = x[p];
        py[u] = y[p];
        pz[u] = z[p];
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const bool valid = base + u * kMeshT + threadIdx.x < n;
      const uint32_t c = valid ? mesh_cell(px[u], py[u], pz[u], g) : 0xffffffffu;
      peers[u] = __match_any_sync(0xffffffffu, c);
      if (valid && lane == (unsigned)(__ffs(peers[u]) - 1))
        slot[u] = atomicAdd(cursor + c, (uint32_t)__popc(peers[u]));
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t p = base + u * kMeshT + threadIdx.x;
      const uint32_t s = __shfl_sync(0xffffffffu, slot[u], __ffs(peers[u]) - 1) +
                         __popc(peers[u] & ((1u << lane) - 1u));
      if (p < n) to.put(s, p, px[u], py[u], pz[u]);
    }
  }
}

// The canonical order: each entry written at its rank among its cell's source
// indices. A warp a cell, up to kCanonSort entries: the keys sorted in
// registers (a bitonic network, 32 K of them for the smallest K that holds the
// cell), left in shared memory, and each entry's key looked up among them. The
// kernel is bound by its instructions: counting the smaller keys one by one is
// two or three a pair, 60 pairs an entry at a mean of 40 a cell. (64.5 M
// particles in 117^3 cells: 0.98 ms counted by a warp a cell, 0.86 by a thread
// an entry, 0.66 sorted.)
constexpr int kCanonT = 256;
constexpr int kCanonSort = 256;    // entries a warp sorts in cell_canon_kernel
constexpr int kCanonLarge = 1024;  // and in cell_canon_large_kernel

// Ascending sort of 32 K values held by one warp, v[j] at index j * 32 + lane:
// partners in other lanes through shuffles, in other registers directly.
template <int K>
__device__ __forceinline__ void warp_sort_keys(uint32_t (&v)[K]) {
  const unsigned lane = threadIdx.x & 31u;
#pragma unroll
  for (int k = 2; k <= 32 * K; k <<= 1) {
#pragma unroll
    for (int d = k >> 1; d > 0; d >>= 1) {
#pragma unroll
      for (int j = 0; j < K; j++) {
        if (d >= 32) {
          const int dj = d >> 5;
          if (j & dj) continue;
          const bool up = ((j << 5) & k) == 0;  // k > 32 here
          const uint32_t a = v[j], b = v[j | dj];
          v[j] = up ? min(a, b) : max(a, b);
          v[j | dj] = up ? max(a, b) : min(a, b);
        } else {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v[j], d);
          const bool up = (((j << 5) | (int)lane) & k) == 0;
          const bool lower = (lane & (unsigned)d) == 0;
          v[j] = lower == up ? min(v[j], o) : max(v[j], o);
        }
      }
    }
  }
}

template <class R>
__device__ __forceinline__ void canon_write(const MeshRec<R>& v, uint32_t dst, R* ox, R* oy, R* oz,
                                            uint32_t* orig) {
  ox[dst] = v.x;
  oy[dst] = v.y;
  oz[dst] = v.z;
  if (orig) orig[dst] = v.i;
}

// One warp orders the cell at [s, e), e - s <= 32 K; keys: 32 K words of its own.
template <int K, class R>
__device__ __forceinline__ void canon_cell(const MeshRec<R>* __restrict__ tmp, uint32_t s, uint32_t e,
                                           uint32_t* keys, R* ox, R* oy, R* oz, uint32_t* orig) {
  const unsigned lane = threadIdx.x & 31u;
  uint32_t v[K], mine[K];
#pragma unroll
  for (int j = 0; j < K; j++) {
    const uint32_t p = s + j * 32 + lane;
    v[j] = mine[j] = p < e ? tmp[p].i : 0xffffffffu;  // above every source index
  }
  warp_sort_keys<K>(v);
#pragma unroll
  for (int j = 0; j < K; j++) keys[j * 32 + lane] = v[j];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < K; j++) {
    const uint32_t p = s + j * 32 + lane;
    if (p < e) {
      uint32_t rank = 0;
#pragma unroll
      for (int step = 16 * K; step > 0; step >>= 1)
        if (keys[rank + step - 1] < mine[j]) rank += step;
      canon_write(tmp[p], s + rank, ox, oy, oz, orig);
    }
  }
  __syncwarp();
}

// One warp orders the cells whose entries, [s, e) together, are no more than its
// lanes: cells k .. k2 - 1 of those whose starts the lanes hold in `first`. Each
// lane's entry finds its cell among the starts and its rank among the lanes of
// the same cell.
template <class R>
__device__ __forceinline__ void canon_few(const MeshRec<R>* __restrict__ tmp, uint32_t s, uint32_t e,
                                          uint32_t first, uint32_t k, uint32_t k2, uint32_t* keys, R* ox,
                                          R* oy, R* oz, uint32_t* orig) {
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t p = s + lane;
  MeshRec<R> v{};
  if (p < e) v = tmp[p];
  keys[lane] = v.i;
  uint32_t c = k;
#pragma unroll
  for (uint32_t step = 16; step > 0; step >>= 1) {
    const uint32_t at = c + step;
    const uint32_t start = __shfl_sync(0xffffffffu, first, at & 31u);
    if (at < k2 && start <= p) c = at;
  }
  const uint32_t begin = __shfl_sync(0xffffffffu, first, c);
  const uint32_t same = __match_any_sync(0xffffffffu, p < e ? c : 0xffffffffu);
  __syncwarp();
  if (p < e) {
    uint32_t rank = 0;
    for (uint32_t m = same; m; m &= m - 1) rank += keys[__ffs(m) - 1] < v.i ? 1u : 0u;
    canon_write(v, begin + rank, ox, oy, oz, orig);
  }
  __syncwarp();
}

// Cells of up to kCanonSort entries, a warp each, or as many neighbours together
// as hold 32 entries between them (a cell at a time 1 M particles in 100^3 cells
// took 0.275 ms a call, now 0.148); the larger ones are listed in `more` (*n_more counts them) for
// cell_canon_large_kernel, which takes four times the registers.
template <class R>
__global__ void __launch_bounds__(kCanonT, 4) cell_canon_kernel(
    const MeshRec<R>* __restrict__ tmp, const uint32_t* __restrict__ offsets,
    uint32_t n_cells_total, R* __restrict__ ox, R* __restrict__ oy, R* __restrict__ oz,
    uint32_t* __restrict__ orig, uint32_t* __restrict__ more, uint32_t* __restrict__ n_more,
    uint32_t span) {
  __shared__ uint32_t keys[kCanonT / 32 * kCanonSort];
  cudaTriggerProgrammaticLaunchCompletion();
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  uint32_t* wk = keys + warp * kCanonSort;
  const uint32_t warps = gridDim.x * (kCanonT / 32);
  // `span` (up to 32) neighbouring cells a warp at a time, their offsets read
  // together.
  for (uint64_t at = (uint64_t)(blockIdx.x * (kCanonT / 32) + warp) * span; at < n_cells_total;
       at += (uint64_t)warps * span) {
    const uint32_t c0 = (uint32_t)at, nc = min(span, n_cells_total - c0);
    const uint32_t first = lane < nc ? offsets[c0 + lane] : 0u;
    const uint32_t next = __shfl_down_sync(0xffffffffu, first, 1);
    const uint32_t end = lane + 1 == nc ? offsets[c0 + nc] : next;  // of lane's cell
    // Past a half warp's entries a cell no two share a warp, and looking for
    // some costs 64.5 M particles in 117^3 cells 1% of the call.
    const bool few = __shfl_sync(0xffffffffu, end, nc - 1) - __shfl_sync(0xffffffffu, first, 0) <= 16u * nc;
    for (uint32_t k = 0; k < nc;) {
      const uint32_t s = __shfl_sync(0xffffffffu, first, k);
      // The cells from the k-th whose entries fit in the warp.
      uint32_t fit = 0;
      if (few) fit = __popc(__ballot_sync(0xffffffffu, lane >= k && lane < nc && end - s <= 32u));
      const uint32_t k2 = k + max(fit, 1u);
      const uint32_t e = __shfl_sync(0xffffffffu, end, k2 - 1), cnt = e - s;
      if (cnt == 0) {
      } else if (fit > 1) {
        canon_few(tmp, s, e, first, k, k2, wk, ox, oy, oz, orig);
      } else if (cnt <= 32) {
        canon_cell<1>(tmp, s, e, wk, ox, oy, oz, orig);
      } else if (cnt <= 64) {
        canon_cell<2>(tmp, s, e, wk, ox, oy, oz, orig);
      } else if (cnt <= 128) {
        canon_cell<4>(tmp, s, e, wk, ox, oy, oz, orig);
      } else if (cnt <= kCanonSort) {
        canon_cell<8>(tmp, s, e, wk, ox, oy, oz, orig);
      } else if (lane == 0) {
        more[atomicAdd(n_more, 1u)] = c0 + k;
      }
      k = k2;
    }
  }
}

// The listed cells: a warp each up to kCanonLarge entries, then the others, the
// CTA's warps together counting each entry's smaller keys as they pass through
// shared memory.
template <class R>
__global__ void __launch_bounds__(kCanonT) cell_canon_large_kernel(
    const MeshRec<R>* __restrict__ tmp, const uint32_t* __restrict__ offsets,
    const uint32_t* __restrict__ more, const uint32_t* __restrict__ n_more, R* __restrict__ ox,
    R* __restrict__ oy, R* __restrict__ oz, uint32_t* __restrict__ orig) {
  __shared__ uint32_t keys[kCanonT / 32 * kCanonLarge];
  cudaGridDependencySynchronize();
  const uint32_t n = *n_more;
  const unsigned warp = threadIdx.x >> 5;
  uint32_t* wk = keys + warp * kCanonLarge;
  for (uint32_t i = blockIdx.x * (kCanonT / 32) + warp; i < n; i += gridDim.x * (kCanonT / 32)) {
    const uint32_t s = offsets[more[i]], e = offsets[more[i] + 1];
    if (e - s <= kCanonLarge / 2)
      canon_cell<16>(tmp, s, e, wk, ox, oy, oz, orig);
    else if (e - s <= kCanonLarge)
      canon_cell<32>(tmp, s, e, wk, ox, oy, oz, orig);
  }
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint32_t s = offsets[more[i]], e = offsets[more[i] + 1];
    if (e - s <= kCanonLarge) continue;
    for (uint32_t p0 = s; p0 < e; p0 += kCanonT) {
      const uint32_t p = p0 + threadIdx.x;
      MeshRec<R> v{};
      if (p < e) v = tmp[p];
      uint32_t rank = 0;
      for (uint32_t k0 = s; k0 < e; k0 += kCanonT / 32 * kCanonLarge) {
        const uint32_t nk = min((uint32_t)(kCanonT / 32 * kCanonLarge), e - k0);
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < nk; k += kCanonT) keys[k] = tmp[k0 + k].i;
        __syncthreads();
#pragma unroll 8
        for (uint32_t k = 0; k < nk; k++) rank += keys[k] < v.i ? 1u : 0u;
      }
      if (p < e) canon_write(v, s + rank, ox, oy, oz, orig);
    }
  }
}

size_t mesh_scratch_bytes(uint64_t n_particles, uint32_t n_cells) {
  const uint64_t cells = (uint64_t)n_cells * n_cells * n_cells;
  return n_particles * sizeof(MeshRec<float>) + (cells + 2) * sizeof(uint32_t) + 1024;
}

template <class R>
static MeshGeom<R> mesh_geom(const DeviceMeshT<R>& m) {
  return MeshGeom<R>{m.n_cells, m.box_length, R(1.0f) / m.cell_length};
}

// cells + 1 counts, then starts and cursors; then how many cells are large.
static uint32_t* mesh_cursor(void* scratch, uint64_t n_particles, size_t record) {
  return (uint32_t*)((char*)scratch + ((n_particles * record + 255) & ~(size_t)255));
}

static unsigned mesh_grid(uint64_t n) {
  return grid_for(n, kMeshT * (n <= kMeshFew ? 1 : kMeshUnroll), 152u * 8u);
}

template <class R>
void mesh_count(const R* x, const R* y, const R* z, uint64_t n_particles, const DeviceMeshT<R>& m,
                void* scratch, cudaStream_t st, const R* bounds, unsigned long long* outside) {
  const uint64_t cells = (uint64_t)m.n_cells * m.n_cells * m.n_cells;
  uint32_t* cursor = mesh_cursor(scratch, n_particles, sizeof(MeshRec<R>));
  SIFG_CUDA(cudaMemsetAsync(cursor, 0, (cells + 2) * sizeof(uint32_t), st));
  if (bounds) SIFG_CUDA(cudaMemsetAsync(outside, 0, sizeof(*outside), st));
  (n_particles <= kMeshFew ? cell_count_kernel<R, 1> : cell_count_kernel<R, kMeshUnroll>)<<<
      mesh_grid(n_particles), kMeshT, 0, st>>>(
      x, y, z, n_particles, mesh_geom(m), cursor, bounds ? bounds[0] : R(0), bounds ? bounds[1] : R(0),
      bounds ? outside : nullptr);
  SIFG_LAUNCH_CHECK();
}

template <class R>
void mesh_build(const R* x, const R* y, const R* z, uint64_t n_particles, DeviceMeshT<R>& m,
                void* scratch, cudaStream_t st, KernelTimer* timer, uint32_t* scan_sums,
                bool canonical, bool counted) {
  const MeshGeom<R> g = mesh_geom(m);
  const uint64_t cells = (uint64_t)m.n_cells * m.n_cells * m.n_cells;
  MeshRec<R>* tmp = (MeshRec<R>*)scratch;
  uint32_t* cursor = mesh_cursor(scratch, n_particles, sizeof(MeshRec<R>));
  if (timer) timer->begin(st);
  if (!counted) mesh_count(x, y, z, n_particles, m, scratch, st, (const R*)nullptr, nullptr);
  exclusive_scan_u32(cursor, (uint32_t)(cells + 1), st, scan_sums);
  SIFG_CUDA(cudaMemcpyAsync(m.offsets, cursor, (cells + 1) * sizeof(uint32_t),
                            cudaMemcpyDeviceToDevice, st));
  auto scatter = [&](auto to) {
    (n_particles <= kMeshFew ? cell_scatter_kernel<R, 1, decltype(to)>
                             : cell_scatter_kernel<R, kMeshUnroll, decltype(to)>)<<<
        mesh_grid(n_particles), kMeshT, 0, st>>>(x, y, z, n_particles, g, cursor, to);
    SIFG_LAUNCH_CHECK();
  };
  if (!canonical) {
    if constexpr (sizeof(R) == 4)
      scatter(ToXyzw{m.xyzw});
    else
      scatter(ToArrays<R>{m.x, m.y, m.z});
    if (timer) timer->end(st);
    m.n_particles = n_particles;
    return;
  }
  scatter(ToRecord<R>{tmp});
  // The scatter's cursors are free: the list of the large cells.
  uint32_t *more = cursor, *n_more = cursor + cells + 1;
  // As many neighbours a warp as still leave every SM its warps.
  const uint32_t span = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(cells / (152u * 64u), 1), 32);
  cell_canon_kernel<R><<<grid_for(cells, kCanonT / 32 * span, 152u * 8u), kCanonT, 0, st>>>(
      tmp, m.offsets, (uint32_t)cells, m.x, m.y, m.z, m.orig, more, n_more, span);
  SIFG_LAUNCH_CHECK();
  // Mostly with nothing to do: launched beside the kernel above, whose end it
  // waits for, so that its launch does not come after (10,000 particles: 3 us).
  cudaLaunchAttribute beside{};
  beside.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  beside.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t large{};
  large.gridDim = (unsigned)std::min<uint64_t>(cells, 152u * 2u);
  large.blockDim = kCanonT;
  large.stream = st;
  large.attrs = &beside;
  large.numAttrs = 1;
  SIFG_CUDA(cudaLaunchKernelEx(&large, cell_canon_large_kernel<R>, (const MeshRec<R>*)tmp,
                               (const uint32_t*)m.offsets, (const uint32_t*)more,
                               (const uint32_t*)n_more, m.x, m.y, m.z, m.orig));
  SIFG_LAUNCH_CHECK();
  if (timer) timer->end(st);
  m.n_particles = n_particles;
}

// ---------------------------------------------------------------------------
// A weighted mesh's columns (chain_mesh.c:800-801, 624-672): each entry's
// weight is the field's at its source index; each cell's weights summed in
// double in mesh order and stored in the form's precision; the total over 64
// fixed blocks of cells, each block's cell sums added in order, the blocks
// then added in order. Every sum in the reference's order, so every bit is
// the reference's.
// ---------------------------------------------------------------------------
template <class R>
__global__ void gather_weights_kernel(const R* __restrict__ fw, const uint32_t* __restrict__ orig,
                                      uint64_t n, R* __restrict__ out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride)
    out[p] = fw[orig[p]];
}

template <class R>
__global__ void cell_weight_kernel(const uint32_t* __restrict__ offsets, const R* __restrict__ w,
                                   uint64_t cells, double* __restrict__ csum, R* __restrict__ cw) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cells; c += stride) {
    double s = 0.0;
    for (uint32_t p = offsets[c]; p < offsets[c + 1]; p++) s = __dadd_rn(s, (double)w[p]);
    csum[c] = s;
    cw[c] = (R)s;
  }
}

constexpr int kWeightBlocks = 64;  // WEIGHT_BLOCKS, chain_mesh.c:642

__global__ void weight_total_kernel(const double* __restrict__ csum, uint64_t cells,
                                    double* __restrict__ total) {
  __shared__ double bt[kWeightBlocks];
  const uint64_t block = (cells + kWeightBlocks - 1) / kWeightBlocks;
  const uint64_t c0 = (uint64_t)threadIdx.x * block;
  const uint64_t c1 = c0 + block < cells ? c0 + block : cells;
  double s = 0.0;
  for (uint64_t c = c0; c < c1; c++) s = __dadd_rn(s, csum[c]);
  bt[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int b = 0; b < kWeightBlocks; b++) t = __dadd_rn(t, bt[b]);
    *total = t;
  }
}

size_t mesh_weights_scratch_bytes(uint32_t n_cells) {
  return (size_t)n_cells * n_cells * n_cells * sizeof(double) + 256;
}

template <class R>
void mesh_weights(const R* field_w, DeviceMeshT<R>& m, void* scratch, double* d_total,
                  cudaStream_t st) {
  const uint64_t cells = (uint64_t)m.n_cells * m.n_cells * m.n_cells;
  gather_weights_kernel<R><<<grid_for(m.n_particles, 256, 152u * 16u), 256, 0, st>>>(
      field_w, m.orig, m.n_particles, m.w);
  SIFG_LAUNCH_CHECK();
  double* csum = (double*)scratch;
  cell_weight_kernel<R><<<grid_for(cells, 128, 152u * 32u), 128, 0, st>>>(m.offsets, m.w, cells,
                                                                         csum, m.cell_w);
  SIFG_LAUNCH_CHECK();
  weight_total_kernel<<<1, kWeightBlocks, 0, st>>>(csum, cells, d_total);
  SIFG_LAUNCH_CHECK();
}

template void mesh_weights<float>(const float*, DeviceMeshT<float>&, void*, double*, cudaStream_t);
template void mesh_weights<double>(const double*, DeviceMeshT<double>&, void*, double*,
                                   cudaStream_t);

template void mesh_build<float>(const float*, const float*, const float*, uint64_t,
                                DeviceMeshT<float>&, void*, cudaStream_t, KernelTimer*, uint32_t*,
                                bool, bool);
template void mesh_build<double>(const double*, const double*, const double*, uint64_t,
                                 DeviceMeshT<double>&, void*, cudaStream_t, KernelTimer*,
                                 uint32_t*, bool, bool);
template void mesh_count<float>(const float*, const float*, const float*, uint64_t,
                                const DeviceMeshT<float>&, void*, cudaStream_t, const float*,
                                unsigned long long*);
template void mesh_count<double>(const double*, const double*, const double*, uint64_t,
                                 const DeviceMeshT<double>&, void*, cudaStream_t, const double*,
                                 unsigned long long*);

}  // namespace sifg
