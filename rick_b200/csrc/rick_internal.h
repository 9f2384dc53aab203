// Internal declarations shared by the librick_b200 translation units.
#pragma once

#include <cuda_runtime.h>
#include <cufft.h>
#include <stdint.h>

#include <atomic>
#include <cmath>

#include "rick_b200.h"

namespace rick {

// Truncated pi of the reference (allvars.h:47, w-stacking.h:6); the w-phase and
// the Gaussian norm use it, and 1e-12 parity needs the same constant.
constexpr double kPi = 3.14159265359;
// Oversampling of the 1-D kernel tables (w-stacking.cu:253).
constexpr int kIncreasePrecision = 5;
// Gaussian width 1/(2 std^2) with std = 1 (w-stacking.cu:254-255).
constexpr double kStd22 = 0.5;
// Edge of a grid tile owned by one gridder work item.
constexpr int kTile = 32;
// Largest supported w_support (odd): footprints fit inside one tile border.
constexpr int kMaxSupport = 15;
// Threads per gridder block.
constexpr int kGridThreads = 256;

// Status plumbing: every internal call returns an int status and records a
// message in thread-local storage.
int set_error(int status, const char *fmt, ...);
int cuda_status(cudaError_t e, const char *what, const char *file, int line);
int cufft_status(cufftResult r, const char *what, const char *file, int line);

#define RICK_CUDA(call)                                                              \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess) return ::rick::cuda_status(e_, #call, __FILE__, __LINE__); \
  } while (0)
#define RICK_CUFFT(call)                                                               \
  do {                                                                                 \
    cufftResult r_ = (call);                                                           \
    if (r_ != CUFFT_SUCCESS) return ::rick::cufft_status(r_, #call, __FILE__, __LINE__); \
  } while (0)
#define RICK_TRY(call)            \
  do {                            \
    int s_ = (call);              \
    if (s_ != RICK_OK) return s_; \
  } while (0)

// Geometry of one imaging job, as the kernels see it.
struct Geometry {
  int nx, ny, nw;       // grid_size_x, grid_size_y, num_w_planes
  int support;          // w_support (odd)
  int half;             // KernelLen = (w_support-1)/2
  int ntx, nty;         // tiles per row / column
  double dx, dw;        // 1/Nx, 1/Nw (init.c:11-12) or as passed to wstack
  double inv_dx, inv_dw; // 1/dx, 1/dw where those are powers of two, else 0 (set_spacing)
  double w_supporth;    // (double)half*dx (init.c:13)
  int select_sector0;   // apply gridding.c:149-188 membership
  int w_first;          // first plane of a w-plane shard (nw planes from here)
  int nw_total;         // planes of the whole cube (0: nw)
  uint64_t nbins() const { return (uint64_t)nw * ntx * nty; }
  // Cell sizes.  A quotient by a power of two is the product with its inverse, to
  // the bit, so the row passes skip the division there.
  void set_spacing(double dx_, double dw_) {
    auto inverse = [](double d) {
      int e = 0;
      return d > 0.0 && std::frexp(d, &e) == 0.5 && e > -1000 && e < 1000 ? 1.0 / d : 0.0;
    };
    dx = dx_;
    dw = dw_;
    inv_dx = inverse(dx_);
    inv_dw = inverse(dw_);
  }
};

// Binned row record (32 bytes: one DRAM sector, one 32-byte load or store).  pu, pv
// are the FP64 pixel positions u/dx, v/dx of w-stacking.cu:143-144; the
// gridder re-derives the cell (int)pos and the fraction pos - (int)pos, exact
// in FP64, so (d + 0.5) - f rounds to the reference's (j + 0.5) - pos exactly.
struct __align__(32) RecF64 {
  double sre, sim;   // sum over channels and polarisations of weight*vis
  double pu, pv;     // pixel position
};

// FP64 sums of a mixed plan's densest tiles: of those with more than kWideParts work
// items (grid.cu).  An FP32 cell loses about sqrt(items / 3) of an add's rounding to the
// items added into it, and larger items lose more in their own 32-bit sums.  Error of
// images against 64 bits, 64^2 on one plane, three array layouts, sources and noise:
// 75,000 rows 1.3, 1.3 and 1.3e-7 (added into FP32 cells 3.1, 3.2 and 4.1e-7 with items
// of 64 records, 3.1, 2.5 and 2.1e-7 with 1024); noise alone 1.7, 1.8 and 1.8e-7 (4.1,
// 3.8 and 4.5e-7 with 64, 18, 17 and 19e-7 with 1024).  The adds of that many items at
// one tile's addresses take longer in FP64 (93 -> 103 us a call; real and imaginary sums
// apart, since interleaved they touch twice the sectors: 126); 300,000 rows on 128^2 x 2
// 145 -> 141.  A tile takes the slot of a hash table that its bin finds first.
constexpr uint32_t kWideParts = 64;
struct WideTiles {
  uint32_t *table = nullptr;  // [slots] bin + 1, or 0: cleared before every gridding
  uint32_t *done = nullptr;   // [slots] items added; 0 between griddings
  double *sums = nullptr;     // [slots][re, im][kTile^2]; 0 between griddings
  uint32_t slots = 0;         // a power of two
};

// Device scratch owned by a plan.
struct Scratch {
  uint32_t *bin_count = nullptr;   // [nbins+1] counts, then exclusive offsets
  uint32_t *bin_cursor = nullptr;  // [nbins]
  uint32_t *item_off = nullptr;    // [nbins+1] work-item offsets
  uint32_t *scan_tmp = nullptr;    // block sums for the scan
  uint64_t *counters = nullptr;    // [8] device counters (see Counter)
  RecF64 *records = nullptr;       // [max_records]
  uint64_t max_records = 0;
  double *table = nullptr;         // 1-D kernel table, 5*support doubles
  WideTiles wide;                  // of a plan in the mixed form
};

// Scratch of the sparse-aware FFT (fft.cu).
struct FftScratch {
  uint32_t *rowmask = nullptr;  // [nw * nty] bit k%32 of word (w, k/32): row k touched
  uint16_t *rowbits = nullptr;  // [nw * ny / 16] the row mask by column-pass thread
  uint32_t *rowlist = nullptr;  // [nw * ny] touched (plane, row) ids
  uint32_t *counts = nullptr;   // [1 + nw] touched rows, then touched rows per plane
  uint32_t *tilemask = nullptr; // [nw * nty * ceil(ntx/32)] bit tx: tile (w, ty, tx) holds records
  void *tw_x = nullptr, *tw_y = nullptr;  // twiddles of the two axes
  void *blocked = nullptr;      // row-transformed planes by column units (cube-sized)
};

// One job of a batch (batch.cu), as the batch kernels see it: the job's
// geometry, its inputs and outputs, and where its slices of the batch-wide
// arrays start.  Work units of every stage are numbered across all jobs; a
// kernel finds the job of a unit by binary search over the unit bases.
struct BatchJob {
  Geometry g;
  int kernel;                      // RICK_KERNEL_*
  int logx, logy;                  // log2 of the axes (sparse FFT sizes)
  uint64_t nrows;                  // rows of the job
  uint32_t nchan, npol;
  int scatter_lanes;               // lanes per row of the sample pass (1, 2, 4, ..., 32)
  int scatter_vec;                 // samples per load of the sample pass (sample_vector)
  uint32_t bin_base;               // first global bin (nw*nty*ntx bins per job)
  uint32_t counts_base;            // first word of the job's [1 + nw] row counts
  uint64_t mask_base;              // first word of the job's row mask [nw * nty]
  uint64_t tile_base;              // first word of the job's tile bitmap [nw * nty * tmw]
  uint64_t list_base;              // first entry of the job's row list [nw * ny]
  const double *uu, *vv, *ww;      // rows (device)
  const float *weight, *vis_re, *vis_im;
  void *cube;                      // [nw][ny][nx] complex (T)
  void *blocked;                   // row transforms by column units (cube-sized)
  const double *table;             // 1-D kernel table (5*support)
  const void *tw_x, *tw_y;         // twiddles of the two axes
  const double *ltab, *mtab;       // phase tables (nx, ny)
  double wmin, dw_phase, dwnorm, norm;
  int phase_on;
  double *img_re, *img_im;         // image (device, [ny][nx])
};

// Batch-wide unit bases of the binning and gridding stages (device arrays of
// njobs + 1 entries, exclusive prefix sums).
struct BatchUnits {
  const uint64_t *row_units;   // 32-row binning units per job
  const uint32_t *bin_base;    // bins per job (== BatchJob::bin_base, plus the total)
};

// FFT stages of a set of jobs (a plan is a set of one): jobs sorted by logx, so
// that the jobs of one row-FFT length are contiguous; the column pass lists them
// grouped by logy.  One launch per FFT length present.
struct FftClass {
  int log;         // log2 of the FFT length
  int lo, hi;      // jobs[lo..hi) (row pass) or col_jobs[lo..hi) (column pass)
  uint32_t units;  // column groups of the class (column pass)
  int planes;      // most planes of a job of the class (column pass)
};
struct FftJobs {
  const BatchJob *jobs = nullptr;    // device [njobs]
  int njobs = 0;
  uint32_t *fft_units = nullptr;     // device [njobs + 1], row-pass units (filled on the device)
  const uint32_t *col_jobs = nullptr;   // device [njobs]
  const uint32_t *col_units = nullptr;  // device [njobs + 1], in col_jobs order
  const uint64_t *mask_base = nullptr;  // device [njobs + 1], row-mask words per job
  uint64_t total_mask_words = 0;
  uint32_t *rowmask = nullptr, *tilemask = nullptr, *rowlist = nullptr, *counts = nullptr;
  uint16_t *rowbits = nullptr;          // two entries per row-mask word
  int cols_parts = 1;                   // blocks a unit's planes are dealt to (one job)
  bool anchored = false;                // factors formed anew along the planes (a batch)
  int n_row_cls = 0, n_col_cls = 0;
  FftClass row_cls[8], col_cls[8];
  // a set of one job (a plan): its host copy; the FFT kernels then take the
  // job as kernel parameters instead of reading the device table
  const BatchJob *one = nullptr;
};

// Transforms (of 2^logn points, 16 values a thread) that a block of the FFT passes
// runs at once (fft_core.cuh, Shape::kGroups).
__host__ __device__ inline int fft_groups_per_block(int logn) {
  const int g = (1 << logn) / 16;
  return g >= 128 ? 1 : 128 / g;
}

enum Counter : int {
  kCntDropped = 0,    // rows outside the cube / sector
  kCntGridded = 1,    // rows that produced records
  kCntRecords = 2,    // records written
  kCntItemNext = 3,   // persistent gridder work counter
  kCntOtherShard = 6, // rows of planes outside the shard
  kNumCounters = 8
};

// Kernel-table construction on the host (w-stacking.cu:35-89).
void make_table(int kernel, int support, double *tab);

// Pipeline stages (bin.cu, grid.cu, phase.cu).
// Both passes expect bin_count [nbins + 1] and bin_cursor [nbins] cleared.
int bin_count_rows(const Geometry &g, uint64_t nrows, const double *uu, const double *vv,
                   const double *ww, Scratch &s, uint32_t max_chunk, cudaStream_t st);
// The samples of all counted rows, or of successive slices of them.
int bin_scatter_rows(const Geometry &g, uint64_t nrows, const double *uu, const double *vv,
                     const double *ww, const float *weight, const float *vis_re,
                     const float *vis_im, uint32_t nchan, uint32_t npol, Scratch &s,
                     cudaStream_t st);
int grid_tiles(const Geometry &g, int kernel, int precision, Scratch &s, void *cube,
               int accumulate, uint32_t max_chunk, cudaStream_t st,
               uint32_t *rowmask = nullptr, uint32_t *tilemask = nullptr);
// Zeroes the tiles that several work items add into (the sparse path does not
// clear the cube).
int zero_split_tiles(const Geometry &g, int precision, Scratch &s, void *cube, cudaStream_t st);
// Sparse-aware FFT (fft.cu).
bool sparse_fft_supported(int nx, int ny);
size_t twiddle_bytes(int n, int precision);
void make_twiddles(int n, int precision, void *tab);  // twiddle_bytes of host memory
void phase_tables(int xaxis, int yaxis, int xaxistot, int yaxistot, double resolution,
                  double *l, double *m);
// Planes w_first .. w_first+nw-1 of an nw_total-plane cube (phase_correction
// with the global plane index; nw_total = nw, w_first = 0 for a whole cube).
int phase_sum(int precision, const void *cube, int xaxis, int yaxis, int nw, int w_first,
              int nw_total, const double *ltab, const double *mtab, double wmin, double wmax,
              double norm, int phase_on, int accumulate, double *img_re, double *img_im,
              cudaStream_t st);
// gridding.c:21-83 on device rows (uvw.cu); scratch: RICK_NORMALIZE_SCRATCH bytes.
int normalize_uvw(uint64_t n, double *uu, double *vv, double *ww, void *scratch,
                  cudaStream_t st);
// counts[0..nbins) -> exclusive offsets in place (counts[nbins] the total) and
// item_off[0..nbins]: exclusive offsets of ceil(count / max_chunk) (scan.cu).
int scan_bins(uint32_t *counts, uint32_t *item_off, uint64_t nbins, uint32_t max_chunk,
              uint32_t *tmp, cudaStream_t st);
uint64_t scan_tmp_words(uint64_t n);

#ifdef __CUDACC__
// Index j of the job that owns unit x: the last j with base[j] <= x, for an
// exclusive prefix base[0..njobs] with x < base[njobs].
template <typename U>
__device__ __forceinline__ int batch_job_of(const U *__restrict__ base, int njobs, U x) {
  int lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (base[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}
#endif

// Batch stages: every job of the batch in one launch per kernel.
// Jobs of one sample-pass schedule (lanes per row, samples per load): entries
// lo..hi-1 of the schedule-ordered job list.
struct ScatterClass {
  int lanes, vec;
  int lo, hi;
  uint64_t units;  // 32-row units of the class
};

struct BatchLaunch {
  const BatchJob *jobs;    // device [njobs]
  int njobs;
  BatchUnits u;
  const uint32_t *sc_jobs;   // device [njobs]: jobs grouped by sample-pass schedule
  const uint64_t *sc_units;  // device [njobs + 1]: 32-row unit prefix in that order
  int n_sc;
  ScatterClass sc[18];
  uint64_t total_row_units;
  uint32_t total_bins;
  int max_support;
  int min_support;
  uint32_t *rowmask, *tilemask;  // batch-wide arrays
  int grid_blocks_per_sm;  // gridder occupancy (tuned)
};
int bin_rows_batch(const BatchLaunch &b, Scratch &s, uint32_t max_chunk, cudaStream_t st);
int grid_tiles_batch(const BatchLaunch &b, int precision, Scratch &s, uint32_t max_chunk,
                     cudaStream_t st);

// The sparse-aware FFT stages (fft.cu) of a set of jobs.  fft_classes fills the
// classes and the host copies of col_jobs / col_units (njobs and njobs + 1
// entries) from the host copy of the jobs (sorted by logx).
void fft_classes(const BatchJob *host_jobs, int njobs, int precision, FftJobs &f,
                 uint32_t *col_jobs, uint32_t *col_units);
// Blocks the planes of one job's column pass are dealt to (FftJobs::cols_parts).
int column_parts(int precision, int nx, int ny, int nw);
int sparse_fft_lists(const FftJobs &f, int precision, cudaStream_t st);  // row lists and row-pass units
int sparse_fft_rows(const FftJobs &f, int precision, cudaStream_t st);
int sparse_fft_cols(const FftJobs &f, int precision, cudaStream_t st);

// The batch internals the serving loop (serve.cu) builds on (batch.cu).
// cols_gate: an event the batch's column pass waits for and records (batches
// launched side by side on several streams), or null.
int batch_create_in(rick_batch **out, const rick_job_desc *jobs, int njobs, int precision,
                    int device, void *arena, uint64_t arena_bytes, const rick_batch_tuning &t,
                    cudaStream_t st, cudaEvent_t cols_gate);
int batch_launch_eager(rick_batch *b, cudaStream_t st);
void batch_destroy(rick_batch *b);
uint64_t batch_bytes(const rick_job_desc *jobs, int njobs, int precision);
bool batch_cached_tuning(int precision, rick_batch_tuning *t);

// Samples per load of the sample pass (4, 2 or 1) for rows of nv samples in npol
// polarisations at these addresses, and the lanes per row for rows of `per_row`
// loads (bin.cu; w-plane shards have schedules of their own there).
int sample_vector(const float *vis_re, const float *vis_im, uint64_t nv, uint32_t npol);
int lanes_per_row(uint64_t per_row);

int num_sms();

// Synchronous copies between host memory (pageable or pinned) and device
// memory; pageable memory goes through a ring of pinned buffers filled and
// drained by a pool of host threads while the copy engine runs (hostcopy.cu).
int copy_to_device(void *dst, const void *src, uint64_t bytes, cudaStream_t st);
int copy_to_host(void *dst, const void *src, uint64_t bytes, cudaStream_t st);

// Kernels launched by this library (reported by rick_launch_count).
extern std::atomic<unsigned long long> g_launches;
#define RICK_LAUNCHED() (::rick::g_launches++)

}  // namespace rick
