// The smoothing stage (smooth.cu).
#pragma once

#include <cufft.h>

#include <memory>
#include <vector>

#include "kernels.cuh"

namespace sifg {

constexpr int kFilterNone = 0;
constexpr int kFilterTopHat = 1;
constexpr int kFilterGaussian = 2;

// Where a smoothing can list the cells it writes at or below a threshold, in
// flat order, by blocks of kBelowBlock cells: block b's entries at the start
// of its region [b * kBelowBlock, (b + 1) * kBelowBlock) of delta and flat,
// their number in counts[b]. counts NULL: no list.
constexpr uint32_t kBelowBlock = 8192;
struct BelowList {
  float thr = 0.f;
  uint32_t* counts = nullptr;  // cells / kBelowBlock
  float* delta = nullptr;      // cells slots
  uint32_t* flat = nullptr;    // cells slots
  // The field itself written too; false where the list is all its reader
  // needs (a run's candidates, under the cell seeds).
  bool field = true;
};

// Window modes: 0 none (SIF_FINDER_KEEP_CIC_WINDOW), 1 full CIC deconvolution,
// 2 aliasing-aware (SIF_FINDER_ALIASING_WINDOW). R is the form's precision:
// float (cuFFT R2C/C2R) or double (D2Z/Z2D).
template <class R>
struct SmootherT {
  uint32_t n = 0;
  R box = 0;
  int window_mode = 1;
  cudaStream_t stream = 0;
  cufftHandle plan_r2c = 0, plan_c2r = 0;  // the plans for n (unset where the transforms are our own)
  DevBuf spectrum, work, lut, win;
  // The plans' work area, one for all of them: they run on `stream`, one at a
  // time. A plan made with its own area would allocate it, and destroying
  // it free it, a device-wide wait that stalls every other engine.
  DevBuf area;
  static constexpr int kLanes = 4;  // smoothings at once, at most
  // Plans by grid size, kept between runs: at most kPlanCache sizes, oldest
  // out; a batch of boxes of many sizes keeps them all.
  static constexpr int kPlanCache = 64;
  struct Plans {
    uint32_t n;
    cufftHandle r2c, c2r;
    size_t work = 0;           // bytes of work area the two need
    void* twiddles = nullptr;  // the own transforms' tables (no plans)
    cufftHandle lane[kLanes - 1] = {};  // the further lanes' inverses, made when first wanted
  };
  size_t plan_work = 0;  // the current plans' need
  // Further lanes, for several smoothings of the one spectrum at once: each a
  // stream with its own inverse plan, transform input, work area and table
  // (lane 0 is `stream` with plan_c2r, work, area and lut).
  struct Lane {
    cudaStream_t st = 0;
    cufftHandle c2r = 0;
    DevBuf work, area, lut;
  };
  Lane extra[kLanes - 1];
  void set_lanes(int lanes, const cudaStream_t* streams);  // after setup
  // The lanes a search at n takes, 1 for `stream` alone: those whose plans are
  // made and one more. A plan and a lane's buffers take most of a millisecond,
  // which one search does not gain, so each of a size's first makes one.
  uint32_t lanes_for(uint32_t n) const;
  const void* twiddles = nullptr;
  std::vector<Plans> plans;
  // The own inverse's filter factors at n = 512, one table per smoothing
  // (filter, radius, sigma, window, box): 257^3 floats (68 MB), the factor of
  // mode (|kx|, |ky|, kz) as the filter pass applies it. Built once, kept
  // (least recently used out past kFactorTables): a run's rungs smooth at the
  // same radii every time.
  struct FactorTable {
    int filter = 0, window_mode = 0;
    R r = 0, sigma = 0, box = 0;
    uint64_t used = 0;
    DevBuf buf;
  };
  static constexpr int kFactorTables = 24;
  std::vector<std::unique_ptr<FactorTable>> factor_tables;
  uint64_t factor_clock = 0;
  const float* factor_table(int filter, R r, R sigma);

  void setup(uint32_t n, R box, int window_mode, cudaStream_t st);
  // grid: n^3 values on the device; with mean set, the density, whose
  // contrast v * (1 / mean) - 1 is transformed (taken as the transform reads
  // it where it can, else in place first).
  void forward(const R* grid, const double* mean = nullptr);
  // Writes the grid smoothed at r (and, with sigma > 0, a Gaussian of sigma
  // on top) into out (n^3 values), asynchronously on the stream.
  // below (float form): the cells at or below below->thr listed as the
  // transform writes them, where lists_below() -- else the caller scans.
  // lane: where it runs (set_lanes; the float form's own transforms only on
  // 0). table: the smoothing's radial table where it is already made, or NULL
  // (the float form's own transforms take none).
  void smooth(int filter, R r, R sigma, R* out, KernelTimer* timer,
              const BelowList* below = nullptr, int lane = 0, const R* table = nullptr);
  // The radial tables of `count` smoothings (sigmas NULL: none on top), each
  // of table_size() values one after another in buf, built on st.
  const R* tables(int filter, const R* radii, const R* sigmas, uint32_t count, DevBuf& buf,
                  cudaStream_t st);
  size_t table_size() const { return 3 * (size_t)(n >> 1) * (n >> 1) + 1; }
  bool lists_below() const { return sizeof(R) == 4 && twiddles != nullptr; }
  void restore(R* out);
  void release();
  ~SmootherT();
};
using Smoother = SmootherT<float>;

// The FP64 form's own transforms (fft64.cu): the sizes they take, their tables
// (for the device), the forward of a grid (with mean set, of its contrast) and
// the inverse of the filtered spectrum through `work`, an n^2 (n / 2 + 1) buffer
// like the spectrum's; `timer` covers the pass that filters.
bool fft64_takes(uint32_t n);
std::vector<double> fft64_tables(uint32_t n);
void fft64_forward(uint32_t n, const double* grid, const double* mean, double2* spec,
                   const double* tab, cudaStream_t st);
void fft64_inverse(uint32_t n, const double2* spec, double2* work, double* out, const double* lut,
                   const double* win, double norm, const double* tab, cudaStream_t st,
                   KernelTimer* timer);

// 1 (default): the own inverse at 512 reads per-smoothing factor tables; 0:
// it evaluates the factors as it applies them. The same bits either way.
void set_factor_tables(int on);

}  // namespace sifg
