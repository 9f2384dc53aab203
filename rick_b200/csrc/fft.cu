// Sparse-aware 2-D inverse FFT of the w-stacked cube, fused with the w-term
// correction and the sum over planes.
//
// fourier_transform.c:34-76 transforms every w-plane with FFTW_BACKWARD and
// scales by 1/(Nx*Ny); phase_correction.cu:191-250 then multiplies each plane by
// its w-phase screen and adds the planes into the image.  A w-plane of a real
// observation holds data on a minority of its rows (the uv tracks of one w
// slice), so here:
//   * the row pass transforms only the rows any footprint touched (a per-tile
//     row mask written by the gridder), reading only the tiles that received
//     records and treating the others as zeros -- so the cube is never cleared;
//   * the column pass loads, for each column, only the touched rows of every
//     plane, transforms the column, and adds the result into per-pixel running
//     sums under the w-correction: the transformed cube is never written back,
//     and the image is written once.
// Both passes run the transforms of fft_core.cuh: 16 values per thread, in FP64
// one row or column per thread group, in the mixed form two at once in packed
// FP32 instructions.  Power-of-two sizes from 64 to 8192; other sizes use the
// cuFFT plan.
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <type_traits>

#include "fft_core.cuh"
#include "rick_internal.h"

namespace rick {

namespace {

using fft::Cx;
using fft::Shape;
using fft::Vec;
using fft::kVpt;

// Grid values (complex) as the gridder wrote them: double2 or float2.
template <typename S> struct CubeVec;
template <> struct CubeVec<double> { using t = double2; };
template <> struct CubeVec<float2> { using t = float2; };

// An element carries one transform in FP64, two in the mixed form: grid rows in
// the row pass; in the column pass, image columns n and n + 1, an element in
// memory being (re, re, im, im) of the two.
using fft::kLanes;

// Row-transformed planes are stored by column units (a unit = one element of
// 16 bytes): element (plane w, row k, unit u) sits at
//   ((w * (units / U) + u / U) * ny + k) * U + u % U,   U = 2,
// 32-byte sectors of two units, consecutive rows next to each other: a column
// pass warp, whose lanes read 32 consecutive rows of one unit, reads 8 lines of
// 128 bytes (a line a lane with whole lines of columns), and the row pass still
// writes whole sectors -- written by halves, 8192-point FP64 rows took 6.7 ms for
// 2.7 (8192^2, 16 planes of 64).
constexpr int kUnitBlock = 2;
__device__ __forceinline__ uint64_t unit_base(uint32_t w, uint32_t u, uint32_t units, int ny) {
  return ((uint64_t)w * (units / kUnitBlock) + u / kUnitBlock) * (uint64_t)ny * kUnitBlock +
         u % kUnitBlock;
}

// The unit of column n (FP64).  Rows of 8192 points are transformed in two
// parts, the even and the odd outputs: their columns are kept apart, so that
// each part writes whole sectors.
__device__ __forceinline__ uint32_t unit_of(uint32_t n, int nx) {
  return nx == 8192 ? (n & 1) * 4096u + (n >> 1) : n;
}

namespace tm {

__device__ __forceinline__ void alloc(uint32_t *smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
// 4 consecutive columns of the thread's lane; the registers are ready after
// wait_ld4, which names them so that no use moves above the wait.
__device__ __forceinline__ void ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void wait_ld4(uint32_t (&a)[4]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3])
               :
               : "memory");
}
// 8 consecutive columns (two pixels' sums, or their steps) of a and of b; the
// registers are ready after wait_ld8x2.
__device__ __forceinline__ void ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void wait_ld8x2(uint32_t (&a)[8], uint32_t (&b)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]),
                 "+r"(a[6]), "+r"(a[7]), "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]),
                 "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7])
               :
               : "memory");
}
// Stores are asynchronous: wait_st before the columns are loaded again.
__device__ __forceinline__ void st4(uint32_t taddr, const uint32_t *r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}
__device__ __forceinline__ void wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

// An element component as the two words of its TMEM columns.
__device__ __forceinline__ void split(double v, uint32_t *w) {
  w[0] = (uint32_t)__double2loint(v);
  w[1] = (uint32_t)__double2hiint(v);
}
__device__ __forceinline__ void split(float2 v, uint32_t *w) {
  w[0] = __float_as_uint(v.x);
  w[1] = __float_as_uint(v.y);
}
template <typename S> __device__ __forceinline__ S join(const uint32_t *w);
template <> __device__ __forceinline__ double join<double>(const uint32_t *w) {
  return __hiloint2double((int)w[1], (int)w[0]);
}
template <> __device__ __forceinline__ float2 join<float2>(const uint32_t *w) {
  return make_float2(__uint_as_float(w[0]), __uint_as_float(w[1]));
}

}  // namespace tm

// ---- Row pass --------------------------------------------------------------------
//
// Inverse FFT along x of the listed touched rows, from the gridded cube into the
// column units.  Tiles that received no record (bit clear in the band's tile
// bitmap) were never written and read as zeros.  A thread group takes one row in
// FP64, two rows of the list in the mixed form (one per lane of its elements);
// at 8192 points, one half of a row's outputs in FP64, one row -- its even and
// odd outputs in the two lanes, which are the two columns of a unit -- mixed.
// Bound by the write of the transformed rows (36,060 rows of 4096: 2.4 GB FP64)
// and, below that, by the load/store pipe: the exchanges and the sector-wide
// stores.  Measured at 4096^2 x 32 / 8192^2: 0.90 / 2.2 ms FP64 (0.93 / 2.7 with
// radix-8 passes and line-wide stores), 0.45 / 1.5 ms mixed (0.63 / 2.1).
template <typename S, int L> struct RowShape {
  using F = Shape<L>;
  static constexpr bool kBothHalves = F::kSplit && kLanes<S> == 2;
  static constexpr int kRows = F::kSplit ? 1 : kLanes<S>;            // rows of a group
  static constexpr int kParts = F::kSplit && kLanes<S> == 1 ? 2 : 1; // groups of a row
};

struct RowSrc {
  uint64_t base;  // the row's first element in the cube
  uint32_t bits;  // bit r: the tile of the thread's input r (x = t + G r) has records
  uint32_t w, k;
  bool active;
};

// Input r (x = t + G r) of the group's rows, as the first loads leave it; row_inputs
// makes the inputs of these.  At 8192 points that takes a second cell (x + N): FP64
// rows read it there (2.74 -> 2.23 ms for 8192^2, 16 planes of 64), the mixed form
// reads both there (1.54 ms for 8192^2 x 32, 1.58 with its cells read early: spills).
template <typename S, int L>
__device__ __forceinline__ Cx<S> row_input(const RowSrc (&src)[kLanes<S>], int t, int r,
                                           const typename CubeVec<S>::t *__restrict__ cube) {
  using F = Shape<L>;
  auto cell = [&](const RowSrc &q, int r) {
    typename CubeVec<S>::t v;
    v.x = 0;
    v.y = 0;
    if ((q.bits >> r) & 1u) v = __ldg(cube + q.base + t + F::G * r);
    return v;
  };
  const auto a = cell(src[0], r);
  if constexpr (kLanes<S> == 2) {
    const auto b = F::kSplit ? cell(src[0], 16 + r) : cell(src[1], r);
    return {make_float2(a.x, b.x), make_float2(a.y, b.y)};
  } else {
    return {a.x, a.y};
  }
}
template <typename S, int L>
__device__ __forceinline__ void row_inputs(const RowSrc (&src)[kLanes<S>], int half, int t,
                                           const typename CubeVec<S>::t *__restrict__ cube,
                                           Cx<S> (&v)[kVpt]) {
  if constexpr (RowShape<S, L>::kBothHalves) {
#pragma unroll
    for (int r = 0; r < kVpt; r++) v[r] = row_input<S, L>(src, t, r, cube);
  }
  if constexpr (Shape<L>::kSplit) {
#pragma unroll
    for (int r = 0; r < kVpt; r++) {
      if constexpr (kLanes<S> == 2) {
        v[r] = {make_float2(v[r].re.x + v[r].re.y, v[r].re.x - v[r].re.y),
                make_float2(v[r].im.x + v[r].im.y, v[r].im.x - v[r].im.y)};
      } else {
        Cx<S> b = {0.0, 0.0};
        if ((src[0].bits >> (16 + r)) & 1u)
          b = fft::unpack(__ldg(cube + src[0].base + t + Shape<L>::G * r + Shape<L>::N));
        v[r] = half ? Cx<S>{v[r].re - b.re, v[r].im - b.im} : Cx<S>{v[r].re + b.re, v[r].im + b.im};
      }
    }
  }
}

// The rows whose inputs v holds: transformed and written.  mid() runs between the
// passes, next(q) when v[q] is written.
template <typename S, int L, typename Mid, typename Next>
__device__ __forceinline__ void fft_row_unit(typename Vec<S>::t *s, const RowSrc (&src)[kLanes<S>],
                                             int half, int t,
                                             typename Vec<S>::t *__restrict__ out, int nx, int ny,
                                             const typename fft::TwVec<S>::t *__restrict__ tw,
                                             Cx<S> (&v)[kVpt], Mid mid, Next next) {
  using F = Shape<L>;
  using RS = RowShape<S, L>;
  constexpr int G = F::G;
  fft::first_pass<L, S>(s, t, RS::kBothHalves ? fft::kBoth : half, v);
  mid();
  if constexpr (RS::kBothHalves) {
    fft::later_passes<L, S>(s, t, [&](int e) { return fft::twiddle(tw + e, tw + F::kTab + e); }, v);
  } else {
    const auto *twh = tw + (F::kSplit && half ? F::kTab : 0);
    fft::later_passes<L, S>(s, t, [&](int e) { return fft::twiddle(twh + e); }, v);
  }
  if constexpr (kLanes<S> == 1) {
    const uint32_t u0 = F::kSplit ? half * F::N + t : t;  // unit_of
    auto *o = out + unit_base(src[0].w, u0, nx, ny) + (uint64_t)src[0].k * kUnitBlock;
#pragma unroll
    for (int q = 0; q < kVpt; q++) {
      if (src[0].active) o[(uint64_t)(G * q) * ny] = fft::pack(v[q]);
      next(q);
    }
  } else if constexpr (RS::kBothHalves) {
    auto *o = out + unit_base(src[0].w, t, nx / 2, ny) + (uint64_t)src[0].k * kUnitBlock;
#pragma unroll
    for (int q = 0; q < kVpt; q++) {
      if (src[0].active) o[(uint64_t)(G * q) * ny] = fft::pack(v[q]);
      next(q);
    }
  } else {
    // columns n, n + 1 are neighbouring lanes' outputs: the even lane takes
    // both for the first row, the odd lane for the second
    const int odd = t & 1;
    const RowSrc r = odd ? src[1] : src[0];
    auto *o = out + unit_base(r.w, (uint32_t)t / 2, nx / 2, ny) + (uint64_t)r.k * kUnitBlock;
#pragma unroll
    for (int q = 0; q < kVpt; q++) {
      const float sr = odd ? v[q].re.x : v[q].re.y, si = odd ? v[q].im.x : v[q].im.y;
      const float gr = __shfl_xor_sync(0xffffffffu, sr, 1), gi = __shfl_xor_sync(0xffffffffu, si, 1);
      const Cx<S> c = odd ? Cx<S>{make_float2(gr, v[q].re.y), make_float2(gi, v[q].im.y)}
                          : Cx<S>{make_float2(v[q].re.x, gr), make_float2(v[q].im.x, gi)};
      if (r.active) {
        // pair-units of a G-aligned step: G/2 units, in blocks of kUnitBlock
        o[(uint64_t)(G / 2 * q) * ny] = fft::pack(c);
      }
      next(q);
    }
  }
}

// Row list entries li, li + 1, ... of a group (a job's arrays): their ids (all bits
// set past the list's end), and the rows these stand for.
template <typename S, int L>
__device__ __forceinline__ void row_ids(uint32_t (&id)[kLanes<S>], uint32_t li, uint32_t nrows,
                                        const uint32_t *__restrict__ rowlist) {
#pragma unroll
  for (int i = 0; i < kLanes<S>; i++)
    id[i] = i < RowShape<S, L>::kRows && li + i < nrows ? __ldg(rowlist + li + i) : ~0u;
}
template <typename S, int L>
__device__ __forceinline__ void row_sources(RowSrc (&src)[kLanes<S>], const uint32_t (&id)[kLanes<S>],
                                            int t, int nx, int ny, int nty, int tmw,
                                            const uint32_t *__restrict__ tilemask) {
  using F = Shape<L>;
#pragma unroll
  for (int i = 0; i < kLanes<S>; i++) {
    RowSrc &r = src[i];
    r.active = id[i] != ~0u;
    const uint32_t rid = r.active ? id[i] : 0;
    r.w = rid / (uint32_t)ny;
    r.k = rid % (uint32_t)ny;
    r.base = ((uint64_t)r.w * ny + r.k) * nx;
    r.bits = 0;
    if (r.active) {
      const uint32_t *tm = tilemask + ((uint64_t)r.w * nty + (r.k >> 5)) * tmw;
      // input r is in tile (t + G r) / 32, a bit of word G r / 1024 (G divides 1024, t < G)
#pragma unroll
      for (int q = 0; q < (F::kSplit ? 32 : 16); q++)
        r.bits |= ((__ldg(tm + (F::G * q >> 10)) >> (((t + F::G * q) >> 5) & 31)) & 1u) << q;
    }
  }
}

// Blocks of the row pass that share an SM: 128 registers a thread.
template <int L> __host__ __device__ constexpr int row_min_blocks() { return 512 / Shape<L>::kThreads; }

// Rows one block of the row pass takes (entries of the row list; a row of 8192
// FP64 points takes two blocks).
template <typename S, int L> __host__ __device__ constexpr int rows_per_block() {
  return Shape<L>::kGroups * RowShape<S, L>::kRows;
}

// One job's row pass (the plan): the job's arrays as kernel parameters.
template <typename S, int L>
__global__ void __launch_bounds__(Shape<L>::kThreads, row_min_blocks<L>())
    k_fft_rows(const typename CubeVec<S>::t *__restrict__ cube, typename Vec<S>::t *__restrict__ out,
               int nx, int ny, int nty, int tmw, const uint32_t *__restrict__ tilemask,
               const uint32_t *__restrict__ rowlist, const uint32_t *__restrict__ counts,
               const typename fft::TwVec<S>::t *__restrict__ tw) {
  using F = Shape<L>;
  using RS = RowShape<S, L>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int grp = threadIdx.x / F::G, t = threadIdx.x % F::G;
  auto *s = reinterpret_cast<typename Vec<S>::t *>(smem_raw) + grp * F::N;
  const uint32_t nrows = counts[0];
  const uint32_t units = (nrows + rows_per_block<S, L>() - 1) / rows_per_block<S, L>() * RS::kParts;
  // a unit's row ids are read during the unit before it and their tile bits between
  // its passes, so that of the three dependent reads only the cells' remains, and
  // those start as the unit's values are written, each into the registers it frees
  // (0.96 -> 0.90 ms FP64, 0.49 -> 0.45 mixed for 36,060 rows of 4096)
  Cx<S> v[kVpt];
  RowSrc src[kLanes<S>], nsrc[kLanes<S>];
  uint32_t id[kLanes<S>];
  auto ids = [&](uint32_t u) {
    row_ids<S, L>(id, u < units ? (u / RS::kParts * F::kGroups + grp) * RS::kRows : nrows, nrows,
                  rowlist);
  };
  auto half_of = [](uint32_t u) { return RS::kParts == 2 ? (int)(u & 1) : 0; };
  ids(blockIdx.x);
  row_sources<S, L>(src, id, t, nx, ny, nty, tmw, tilemask);
#pragma unroll
  for (int r = 0; r < kVpt; r++)
    if (!RS::kBothHalves) v[r] = row_input<S, L>(src, t, r, cube);
  for (uint32_t u = blockIdx.x; u < units;) {
    const uint32_t un = u + gridDim.x;
    row_inputs<S, L>(src, half_of(u), t, cube, v);
    ids(un);
    fft_row_unit<S, L>(
        s, src, half_of(u), t, out, nx, ny, tw, v,
        [&] { row_sources<S, L>(nsrc, id, t, nx, ny, nty, tmw, tilemask); },
        [&](int q) {
          if (!RS::kBothHalves) v[q] = row_input<S, L>(nsrc, t, q, cube);
        });
#pragma unroll
    for (int i = 0; i < kLanes<S>; i++) src[i] = nsrc[i];
    u = un;
  }
}

// Row pass over the jobs lo..hi-1 of a batch (all of FFT length 2^L along x): the
// row-pass units of job j (blocks' worth of touched rows) are fft_units[j] ..
// fft_units[j+1]-1.
template <typename S, int L>
__global__ void __launch_bounds__(Shape<L>::kThreads, row_min_blocks<L>())
    k_fft_rows_multi(const BatchJob *__restrict__ jobs, int lo, int hi,
                     const uint32_t *__restrict__ fft_units, const uint32_t *__restrict__ tilemask,
                     const uint32_t *__restrict__ rowlist, const uint32_t *__restrict__ counts) {
  using F = Shape<L>;
  using V = typename Vec<S>::t;
  using RS = RowShape<S, L>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int grp = threadIdx.x / F::G, t = threadIdx.x % F::G;
  V *s = reinterpret_cast<V *>(smem_raw) + grp * F::N;
  const uint32_t u1 = fft_units[hi];
  for (uint32_t u = fft_units[lo] + blockIdx.x; u < u1; u += gridDim.x) {
    const int j = lo + batch_job_of(fft_units + lo, hi - lo, u);
    const BatchJob &J = jobs[j];
    uint32_t id[kLanes<S>];
    RowSrc src[kLanes<S>];
    row_ids<S, L>(id, ((u - fft_units[j]) * F::kGroups + grp) * RS::kRows, counts[J.counts_base],
                  rowlist + J.list_base);
    row_sources<S, L>(src, id, t, J.g.nx, J.g.ny, J.g.nty, (J.g.ntx + 31) / 32,
                      tilemask + J.tile_base);
    Cx<S> v[kVpt];
#pragma unroll
    for (int r = 0; r < kVpt; r++)
      if (!RS::kBothHalves) v[r] = row_input<S, L>(src, t, r, (const typename CubeVec<S>::t *)J.cube);
    row_inputs<S, L>(src, 0, t, (const typename CubeVec<S>::t *)J.cube, v);
    fft_row_unit<S, L>(s, src, 0, t, (V *)J.blocked, J.g.nx, J.g.ny,
                       (const typename fft::TwVec<S>::t *)J.tw_x, v, [] {}, [](int) {});
  }
}

// ---- Column pass -----------------------------------------------------------------
//
// Each thread group owns one unit (an image column in FP64, columns n and n + 1
// in the mixed form) and walks the planes with data in decreasing w, with the
// w-correction as a Horner recurrence: with s = exp(i 2 pi dw (root - 1)) the
// per-pixel factor between consecutive planes and
// P = dwnorm root exp(i 2 pi wterm_lo (root - 1)) that of the lowest plane with
// data,
//     image = P * (((x_hi s^g + ...) s^g' + x_lo)
// so each pixel carries two complex values across planes -- its running sum and
// its step s -- and the phase needs one sincos per pixel for s and one for P per
// column, none per plane.  The reference evaluates every plane's factor with its
// own sincos (phase_correction.cu:205-226); the recurrence's products move each
// factor by a few ulp per plane.  Modelled in long double for the worst pixels:
// 8.4e-14 at 4096^2 x 32 planes (w from -7.5e3 to 7.8e3 wavelengths) and 2.6e-13
// at 8192^2 x 64 planes (w to 1.1e5), below the rounding of the reference's own
// per-plane phase argument there (1.3e-13 and 3.3e-13 at the image corner).  The
// mixed form's sums and steps are FP32 (their arguments and sincos FP64): the
// FP32 recurrence adds ~4e-7 relative error over 32 planes, within the FP32
// transform's own.
//
// The two complex values (eight 32-bit words a pixel in either form) live in
// tensor memory (TMEM, 512 columns x 128 lanes of 32 bits per SM), not in
// registers: the thread's 16 values of the transform take 64 registers, so 512
// threads share an SM (two 4096-point columns, four blocks of shorter ones),
// which is what TMEM holds, too.  Bounds per plane and 4096-point unit: FP64 (or
// packed FP32) issue 2,600 cycles of a sub-partition, load/store pipe ~3,600 of
// the SM (two exchanges 2,048, a wavefront per touched row ~1,130, the image);
// with 16 warps an SM the two overlap in part: 5,300 measured.  With the finish, against
// two columns a block in radix-8 passes: 3.42 -> 2.49 ms FP64 and 2.55 -> 1.29 mixed
// (4096^2 x 32), 10.5 -> 6.6 ms FP64 (8192^2, 16 planes of 64) and 10.9 -> 6.3
// mixed (8192^2 x 32).  Warp w of a block reaches lanes 32 (w % 4) ..
// +31 (its lane quarter); the warps of one quarter split its columns.

// The type of the sums and steps: FP64; FP32 in the mixed form from 1024-point
// columns on (shorter ones keep FP64 sums and steps for each of a unit's two
// columns, twice the words).
template <typename S, int L> struct ColState {
  static constexpr bool kWide = kLanes<S> == 2 && L <= 9;
  static constexpr int kSlots = kWide ? 2 : 1;            // state values of 4 words a pixel
  static constexpr uint32_t kStepCol = 4 * kVpt * kSlots; // TMEM columns of a thread's sums
  using T = std::conditional_t<kWide, double, S>;
};

// Where the sums take the steps of planes without data: pixel by pixel in the loop that
// adds a plane, or in a loop of its own before it.  The former makes the unrolled loop
// long, and with few warps an SM it runs at the rate its instructions are fetched (us,
// in the loop and apart: one mixed job of 64^2 x 64 planes 265 and 163, of 512^2 x 64
// 353 and 250, 24 of them 2,969 and 2,352; column pass of 4096^2 x 32 FP64 2,586 and
// 2,519, of 8192^2 x 32 mixed 6,687 and 6,320); but the packed FP32 state of columns of
// 1024 to 4096 points spills with the second (4096^2 x 32 mixed 1,303 and 1,357).
template <typename S, int L> constexpr bool kGapInLoop = kLanes<S> == 2 && L >= 10 && L <= 12;

// From 1024-point columns on the column pass leaves the sums, unit by unit, in the
// gridded cube, which the row pass has read, and k_fft_finish applies P and turns
// them into image rows.  Written by the column pass itself the image rows of a unit
// are pieces of 8 or 16 bytes, a whole 32-byte sector of traffic each, and its last
// warps compute P with little else in flight.  Column pass and finish, both ways:
// 0.49 -> 0.23 ms FP64 and 0.36 -> 0.14 mixed (4096^2, one plane), 2.88 -> 0.99 and
// 2.38 -> 0.63 (8192^2, one plane), 1.40 -> 1.31 ms mixed (4096^2 x 32), 7.2 -> 6.9 FP64
// (8192^2 x 16 of 64).  Clusters of blocks that write whole sectors together were
// slower, 3.9 ms for the 2.64 of 4096^2 x 32: with TMEM in use one block of a cluster
// launch fits an SM.  The sums keep their type; a unit's row takes 16 bytes, a plane
// of the cube in either form.  (Wide sums do not fit; their short columns lie side by
// side in a block, so that their pieces meet in L2.)
template <int L> constexpr bool kFinish = L >= 10;

// The per-job inputs of the column pass.
template <typename S> struct ColJob {
  const typename Vec<S>::t *cube;  // row transforms by column units
  int nx, ny, nw;
  int w_first, nw_total;           // w-plane shard: global index of local plane 0, cube planes
  const uint16_t *rowbits;         // [nw * ny / 16]: rows t + G r of a plane as bit r of entry t
  const uint32_t *counts;          // [1 + nw]
  const typename fft::TwVec<S>::t *tw;  // twiddles of the y axis
  const double *ltab, *mtab;
  double wmin, dw, dwnorm, norm;
  int phase_on;
  int anchor;                      // planes of a group with a factor of its own (kAnchored)
  double *img_re, *img_im;
  typename Vec<S>::t *sums;        // [units][ny], L = 13: [units][half][ny / 2] (kFinish, groups)
};

// The column pass of a batch whose schedule asks for it (planes_in_flight 1 or 2, a
// server's) sums groups of kAnchorPlanes planes by themselves, each group's factor
// formed anew from its lowest plane: the steps' rounding otherwise adds up over all
// planes.  Off the 64-bit image in one sum / by groups: mixed 1024^2 x 64 planes 7.1e-7 /
// 2.6e-7 (one job 394 / 511 us), 2048^2 x 24 3.6e-7 / 2.7e-7 (473 / 563 us); FP64 1024^2
// x 16 1.5e-14 / 1.0e-14 (257 / 267 us), 512^2 x 64 7.4e-15 / 4.5e-15 (281 / 357 us).
// FP32 sums of up to kPlainPlanes planes are left whole: the transforms' own error is
// the larger there.
constexpr int kAnchorPlanes = 8, kPlainPlanes = 16;
template <typename S, int L> constexpr bool kAnchored = kLanes<S> == 1 || L >= 10;
template <typename S> __host__ __device__ constexpr int plain_planes() {
  return kLanes<S> == 1 ? kAnchorPlanes : kPlainPlanes;
}

// sum += total * (factor of plane `from` / factor of plane `to`) for one pixel with root
// minus one rm1 (of each lane): the sum of the groups above, down to plane `from`, joins
// that of the group whose lowest plane is `to`.
template <typename S>
__device__ __forceinline__ void join_groups(uint32_t *sum, Cx<S> total, const ColJob<S> &J, int from,
                                            int to, const double (&rm1)[kLanes<S>]) {
  const double twopi = 2.0 * kPi;
  auto turn = [&](int w, double rootm1) {
    return __dmul_rn(__dmul_rn(twopi, __dadd_rn(J.wmin, __dmul_rn((double)(J.w_first + w), J.dw))),
                     rootm1);
  };
  double er[kLanes<S>], ei[kLanes<S>];
#pragma unroll
  for (int c = 0; c < kLanes<S>; c++) {
    // the difference of the two rounded arguments, and what it leaves (two-sum)
    const double a = turn(from, rm1[c]), b = turn(to, rm1[c]);
    const double d = __dsub_rn(a, b), bb = __dsub_rn(a, d);
    const double rest = __dsub_rn(__dsub_rn(a, __dadd_rn(d, bb)), __dsub_rn(b, bb));
    double sn, cs;
    sincos(d, &sn, &cs);
    er[c] = fma(-rest, sn, cs);
    ei[c] = fma(rest, cs, sn);
  }
  const S ar = tm::join<S>(sum), ai = tm::join<S>(sum + 2);
  if constexpr (kLanes<S> == 2) {
    const auto re = [](double x, double y, double c, double s, double a) { return (float)fma(x, c, fma(-y, s, a)); };
    const auto im = [](double x, double y, double c, double s, double a) { return (float)fma(x, s, fma(y, c, a)); };
    tm::split(make_float2(re(total.re.x, total.im.x, er[0], ei[0], ar.x),
                          re(total.re.y, total.im.y, er[1], ei[1], ar.y)), sum);
    tm::split(make_float2(im(total.re.x, total.im.x, er[0], ei[0], ai.x),
                          im(total.re.y, total.im.y, er[1], ei[1], ai.y)), sum + 2);
  } else {
    tm::split(fma(total.re, er[0], fma(-total.im, ei[0], ar)), sum);
    tm::split(fma(total.re, ei[0], fma(total.im, er[0], ai)), sum + 2);
  }
}

// Unit u of one job, column u or columns 2u, 2u + 1 (with L = 13, half `half` of
// its pixels), over the planes lo..hi-1, by the group's thread t; the result is
// stored in the image, or (add) added to it.  taddr: the thread's TMEM address,
// pixel q's sum at 4 q (wide state: at 8 q, column by column) and its step kStepCol
// further.
template <typename S, int L, bool ANCHOR = false>
__device__ __forceinline__ void fft_col_unit(typename Vec<S>::t *s, uint32_t u, int half, int lo,
                                             int hi, bool add, int t, const ColJob<S> &J,
                                             uint32_t taddr) {
  using F = Shape<L>;
  using V = typename Vec<S>::t;
  using CS = ColState<S, L>;
  using A = typename CS::T;
  constexpr int G = F::G, NL = kLanes<S>, M = CS::kSlots;
  constexpr uint32_t kStepCol = CS::kStepCol;
  const int ny = J.ny;
  const uint32_t units = (uint32_t)J.nx / NL;
  const uint32_t *__restrict__ counts = J.counts;
  const bool phase = J.phase_on && J.nw_total > 1;
  const double twopi = 2.0 * kPi;  // exact doubling of the reference's pi
  auto prev_plane = [&](int iw) {   // planes without data add exact zeros
    do { iw--; } while (iw >= lo && __ldg(counts + 1 + iw) == 0);
    return iw;
  };
  // bit r: whether row t + G r of plane iw was touched (L = 13: bit 16 + r for
  // row t + G r + N)
  auto row_bits = [&](int iw) {
    const uint16_t *p = J.rowbits + (uint64_t)iw * (ny / 16) + t;
    uint32_t b = __ldg(p);
    if (F::kSplit) b |= (uint32_t)__ldg(p + G) << 16;
    return b;
  };
  const uint32_t mu = NL == 1 ? unit_of(u, J.nx) : u;
  auto plane_rows = [&](int iw) { return J.cube + unit_base(iw, mu, units, ny) + t * kUnitBlock; };
  auto row = [&](const V *col, uint32_t bits, int r) {  // row t + G r (r >= 16: + N)
    Cx<S> v = {fft::splat<S>(0.0), fft::splat<S>(0.0)};
    if ((bits >> r) & 1u) v = fft::unpack(__ldg(col + r * G * kUnitBlock));
    return v;
  };
  // sqrt(1 - l^2 - m^2), phase_correction.cu:56-64
  auto pixel_row = [&](int q) {
    const int m = t + G * q;
    return F::kSplit ? 2 * m + half : m;
  };
  auto root_of = [](double l, double mm) {
    return __dsqrt_rn(__dsub_rn(1.0, __dadd_rn(__dmul_rn(l, l), __dmul_rn(mm, mm))));
  };
  int iw = prev_plane(hi);
  if (iw < lo) {  // no data at all
    if (add || kFinish<L>) return;
#pragma unroll
    for (int q = 0; q < kVpt; q++)
      for (int c = 0; c < NL; c++) {
        const uint64_t o = (uint64_t)pixel_row(q) * J.nx + NL * u + c;
        J.img_re[o] = 0.0;
        J.img_im[o] = 0.0;
      }
    return;
  }
  int nxt = prev_plane(iw);
  // sums (zero) and steps (not used by a single plane) into TMEM
  const double dwstep = __dmul_rn(twopi, J.dw);
  auto set_state = [&](int q, const double (&cs)[NL], const double (&sn)[NL]) {
#pragma unroll
    for (int c = 0; c < M; c++) {
      Cx<A> st;
      if constexpr (kLanes<A> == 2)
        st = {make_float2((float)cs[0], (float)cs[1]), make_float2((float)sn[0], (float)sn[1])};
      else
        st = {cs[c], sn[c]};
      uint32_t z4[4] = {0, 0, 0, 0}, w4[4];
      tm::split(st.re, w4);
      tm::split(st.im, w4 + 2);
      tm::st4(taddr + 4 * (M * q + c), z4);
      tm::st4(taddr + kStepCol + 4 * (M * q + c), w4);
    }
  };
  double l[NL], mm = 0.0, cs[NL], sn[NL];
#pragma unroll
  for (int i = 0; i < NL; i++) {
    cs[i] = 1.0;
    sn[i] = l[i] = 0.0;
  }
  if (phase && nxt >= lo) {
    // (a pixel's m is read while the one before it is worked on)
    mm = J.mtab[pixel_row(0)];
#pragma unroll
    for (int i = 0; i < NL; i++) l[i] = J.ltab[NL * u + i];
#pragma unroll 1
    for (int q = 0; q < kVpt; q++) {
      const double mm_next = J.mtab[pixel_row(min(q + 1, kVpt - 1))];
#pragma unroll
      for (int i = 0; i < NL; i++)
        sincos(__dmul_rn(dwstep, __dsub_rn(root_of(l[i], mm), 1.0)), &sn[i], &cs[i]);
      set_state(q, cs, sn);
      mm = mm_next;
    }
  } else {
#pragma unroll 1
    for (int q = 0; q < kVpt; q++) set_state(q, cs, sn);
  }
  const auto *tw = J.tw + (F::kSplit && half ? F::kTab : 0);
  // the rows a first pass takes: with L = 13, t + G r and t + G r + N combined
  auto combine = [&](Cx<S> lo, Cx<S> hi) {
    return half ? Cx<S>{fft::sub(lo.re, hi.re), fft::sub(lo.im, hi.im)}
                : Cx<S>{fft::add(lo.re, hi.re), fft::add(lo.im, hi.im)};
  };
  Cx<S> v[kVpt];
  uint32_t bits = row_bits(iw);
  const V *col = plane_rows(iw);
#pragma unroll
  for (int r = 0; r < kVpt; r++) {
    v[r] = row(col, bits, r);
    if constexpr (F::kSplit) v[r] = combine(v[r], row(col, bits, 16 + r));
  }
  // the next plane and its row bits are found a plane ahead: a warp that needs
  // them does not wait for the loads
  uint32_t nbits = nxt >= lo ? row_bits(nxt) : 0u;
  int prev = iw;
  tm::wait_st();
  // ANCHOR: the sum of the groups done, in the place of the job's column sums
  V *total = J.sums + (uint64_t)u * ny + t;
  int lowest = lo, done = -1;  // done: lowest plane of the groups in `total`
  if constexpr (ANCHOR)
    while (__ldg(counts + 1 + lowest) == 0) lowest++;
  auto joined = [&](int q, uint32_t (&sum)[4], int to) {
    double rm1[NL];
#pragma unroll
    for (int c = 0; c < NL; c++)
      rm1[c] = __dsub_rn(root_of(J.ltab[NL * u + c], J.mtab[pixel_row(q)]), 1.0);
    join_groups<S>(sum, fft::unpack(total[G * q]), J, done, to, rm1);
  };
  for (;;) {
    col = plane_rows(nxt >= lo ? nxt : iw);
    const int nxt2 = nxt >= lo ? prev_plane(nxt) : nxt;
    const uint32_t nbits2 = nxt2 >= lo ? row_bits(nxt2) : 0u;
    // the index is made opaque here, so that the shared-memory addresses of the
    // passes are formed where they are used and not held (spilled) across planes
    int tp = t;
    asm volatile("" : "+r"(tp));
    fft::first_pass<L, S>(s, tp, half, v);
    if constexpr (ANCHOR) {
      if (phase && (prev - lowest) / J.anchor != (iw - lowest) / J.anchor) {
        // plane prev was the lowest of its group (no values are held here)
#pragma unroll 1
        for (int q = 0; q < kVpt; q++) {
          uint32_t sum[4], zero[4] = {0, 0, 0, 0};
          tm::ld4(taddr + 4 * q, sum);
          tm::wait_ld4(sum);
          tm::st4(taddr + 4 * q, zero);
          if (done >= 0) joined(q, sum, prev);
          total[G * q] = fft::pack(Cx<S>{tm::join<S>(sum), tm::join<S>(sum + 2)});
        }
        tm::wait_st();
        done = prev;
      }
    }
    // planes without data in between: sum * step^(gap - 1) (while no values are held)
    const int gap = prev - iw;
    if (!kGapInLoop<S, L> && gap > 1) {
#pragma unroll 1
      for (int i0 = 0; i0 < kVpt * M; i0 += 2) {
        uint32_t sum[8], step[8];
        tm::ld8(taddr + 4 * i0, sum);
        tm::ld8(taddr + kStepCol + 4 * i0, step);
        tm::wait_ld8x2(sum, step);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          A ar = tm::join<A>(sum + 4 * h), ai = tm::join<A>(sum + 4 * h + 2);
          const A sr = tm::join<A>(step + 4 * h), si = tm::join<A>(step + 4 * h + 2);
#pragma unroll 1
          for (int g2 = 1; g2 < gap; g2++) {
            const A tr = fft::fma_(ar, sr, fft::neg(fft::mul(ai, si)));
            ai = fft::fma_(ar, si, fft::mul(ai, sr));
            ar = tr;
          }
          tm::split(ar, sum + 4 * h);
          tm::split(ai, sum + 4 * h + 2);
        }
        tm::st8(taddr + 4 * i0, sum);
      }
      tm::wait_st();
    }
    fft::later_passes<L, S>(
        s, tp, [&](int e) { return fft::twiddle(tw + e); }, v);
    // sum = sum * step^gap + x, two pixels at a time; as their values are
    // consumed, the next plane's rows take their registers (more pixels per
    // TMEM access, or the next pair's access ahead, spill registers: 2.62 ms at
    // 4096^2 x 32 FP64 against 2.86 and more)
#pragma unroll
    for (int i0 = 0; i0 < kVpt * M; i0 += 2) {
      uint32_t sum[8], step[8];
      tm::ld8(taddr + 4 * i0, sum);
      tm::ld8(taddr + kStepCol + 4 * i0, step);
      tm::wait_ld8x2(sum, step);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int q = (i0 + h) / M;
        Cx<A> x;
        if constexpr (CS::kWide)
          x = h ? Cx<A>{(double)v[q].re.y, (double)v[q].im.y}
                : Cx<A>{(double)v[q].re.x, (double)v[q].im.x};
        else
          x = v[q];
        A ar = tm::join<A>(sum + 4 * h), ai = tm::join<A>(sum + 4 * h + 2);
        const A sr = tm::join<A>(step + 4 * h), si = tm::join<A>(step + 4 * h + 2);
        if constexpr (kGapInLoop<S, L>) {
          for (int g2 = 1; g2 < gap; g2++) {  // planes without data in between
            const A tr = fft::fma_(ar, sr, fft::neg(fft::mul(ai, si)));
            ai = fft::fma_(ar, si, fft::mul(ai, sr));
            ar = tr;
          }
        }
        tm::split(fft::fma_(ar, sr, fft::fma_(fft::neg(ai), si, x.re)), sum + 4 * h);
        tm::split(fft::fma_(ar, si, fft::fma_(ai, sr, x.im)), sum + 4 * h + 2);
        if constexpr (!F::kSplit || NL == 2)
          if (M == 1 || h == 1) v[q] = row(col, nbits, q);
      }
      tm::st8(taddr + 4 * i0, sum);
    }
    if constexpr (F::kSplit) {
#pragma unroll
      for (int q = 0; q < kVpt; q++) {  // (FP64 spills with the first rows read earlier)
        if constexpr (NL == 1) v[q] = row(col, nbits, q);
        v[q] = combine(v[q], row(col, nbits, 16 + q));
      }
    }
    tm::wait_st();
    prev = iw;
    if (nxt < lo) break;
    iw = nxt;
    nxt = nxt2;
    nbits = nbits2;
  }
  if constexpr (kFinish<L>) {
    if (!add) {
      V *to = J.sums + (uint64_t)u * ny + half * F::N + t;
#pragma unroll 4
      for (int q = 0; q < kVpt; q++) {
        uint32_t a4[4];
        tm::ld4(taddr + 4 * q, a4);
        tm::wait_ld4(a4);
        if constexpr (ANCHOR) {
          if (done >= 0) joined(q, a4, prev);
        }
        to[G * q] = fft::pack(Cx<S>{tm::join<S>(a4), tm::join<S>(a4 + 2)});
      }
      return;
    }
  }
  // image = norm * P * sum, P the factor of the lowest plane with data
  const double cw = __dmul_rn(twopi, __dadd_rn(J.wmin, __dmul_rn((double)(J.w_first + prev), J.dw)));
  const bool vec = NL == 2 && ((reinterpret_cast<uintptr_t>(J.img_re) |
                                reinterpret_cast<uintptr_t>(J.img_im)) & 15u) == 0;
  mm = phase ? J.mtab[pixel_row(0)] : 0.0;
#pragma unroll
  for (int c = 0; c < NL; c++) l[c] = phase ? J.ltab[NL * u + c] : 0.0;
#pragma unroll 1
  for (int q = 0; q < kVpt; q++) {
    const double mm_next = phase ? J.mtab[pixel_row(min(q + 1, kVpt - 1))] : 0.0;
    double re[NL], im[NL];
#pragma unroll
    for (int c = 0; c < NL; c++) {
      double ar, ai;
      uint32_t a4[4];
      tm::ld4(taddr + 4 * (M * q + (CS::kWide ? c : 0)), a4);
      tm::wait_ld4(a4);
      if constexpr (ANCHOR) {
        if (done >= 0) joined(q, a4, prev);
      }
      const A sr = tm::join<A>(a4), si = tm::join<A>(a4 + 2);
      if constexpr (kLanes<A> == 2) {
        ar = c ? sr.y : sr.x;
        ai = c ? si.y : si.x;
      } else {
        ar = sr;
        ai = si;
      }
      double pr = 1.0, pi = 0.0;
      if (phase) {
        const double root = root_of(l[c], mm);
        double sn, cs;
        sincos(__dmul_rn(cw, __dsub_rn(root, 1.0)), &sn, &cs);
        const double amp = J.dwnorm * root;
        pr = cs * amp;
        pi = sn * amp;
      }
      re[c] = J.norm * fma(ar, pr, -ai * pi);
      im[c] = J.norm * fma(ar, pi, ai * pr);
    }
    const uint64_t o = (uint64_t)pixel_row(q) * J.nx + NL * u;
    if (add) {
#pragma unroll
      for (int c = 0; c < NL; c++) {
        atomicAdd(J.img_re + o + c, re[c]);
        atomicAdd(J.img_im + o + c, im[c]);
      }
    } else if (vec) {
      *reinterpret_cast<double2 *>(J.img_re + o) = make_double2(re[0], re[NL - 1]);
      *reinterpret_cast<double2 *>(J.img_im + o) = make_double2(im[0], im[NL - 1]);
    } else {
#pragma unroll
      for (int c = 0; c < NL; c++) {
        J.img_re[o + c] = re[c];
        J.img_im[o + c] = im[c];
      }
    }
    mm = mm_next;
  }
}

// TMEM columns of a thread (16 pixels of 8 words, 16 in the wide state) and of a
// block: a thread's per warp of a lane quarter.
template <typename S, int L> __host__ __device__ constexpr uint32_t thread_tm_columns() {
  return 2 * ColState<S, L>::kStepCol;
}
template <typename S, int L> __host__ __device__ constexpr uint32_t col_tm_columns() {
  return (uint32_t)(Shape<L>::kThreads / 128) * thread_tm_columns<S, L>();
}
// Blocks that share an SM: as many as its 512 TMEM columns hold (128 registers a
// thread).
template <typename S, int L> __host__ __device__ constexpr int col_blocks() {
  return (int)(512u / col_tm_columns<S, L>());
}
template <int L> __host__ __device__ constexpr size_t col_smem_bytes() { return (size_t)Shape<L>::kThreads * kVpt * 16 + 16; }

// A block's TMEM: allocated by its first warp, addressed by every thread.
template <typename S, int L> struct BlockTmem {
  uint32_t base, addr;
  __device__ __forceinline__ explicit BlockTmem(uint32_t *slot) {
    const int warp = threadIdx.x / 32;
    if (warp == 0) {
      tm::alloc(slot, col_tm_columns<S, L>());
      tm::relinquish();
    }
    tm::fence_before();
    __syncthreads();
    tm::fence_after();
    base = *slot;
    addr = base + ((uint32_t)(32 * (warp % 4)) << 16) + (uint32_t)(warp / 4) * thread_tm_columns<S, L>();
  }
  __device__ __forceinline__ void release() {
    tm::fence_before();
    __syncthreads();
    if (threadIdx.x / 32 == 0) {
      tm::fence_after();
      tm::dealloc(base, col_tm_columns<S, L>());
    }
  }
};

// One job's column pass: units over a persistent grid (L = 13: the halves of a
// unit are neighbouring blocks' work, and read the same rows).  parts > 1: the
// planes are dealt to that many blocks, which add into the cleared image.
template <typename S, int L>
__global__ void __launch_bounds__(Shape<L>::kThreads, col_blocks<S, L>()) k_fft_cols(ColJob<S> J, int parts) {
  using F = Shape<L>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int grp = threadIdx.x / F::G, t = threadIdx.x % F::G;
  auto *s = reinterpret_cast<typename Vec<S>::t *>(smem_raw) + grp * F::N;
  BlockTmem<S, L> tmem(reinterpret_cast<uint32_t *>(smem_raw + col_smem_bytes<L>() - 16));
  constexpr int kParts = F::kSplit ? 2 : 1;
  const uint32_t nb = (uint32_t)J.nx / kLanes<S> / F::kGroups * kParts;
  for (uint32_t b = blockIdx.x; b < nb * parts; b += gridDim.x) {
    const uint32_t ub = b / parts, part = b % parts;
    fft_col_unit<S, L>(s, ub / kParts * F::kGroups + grp, (int)(ub % kParts),
                       (int)((uint64_t)part * J.nw / parts), (int)((uint64_t)(part + 1) * J.nw / parts),
                       parts > 1, t, J, tmem.addr);
  }
  tmem.release();
}

// The column pass over the jobs col_jobs[lo..hi-1] of a batch (all of FFT length
// 2^L along y): the blocks' worths of units of the k-th listed job are
// col_units[k] .. col_units[k+1]-1.  ANCHOR: factors formed anew (kAnchored).
template <typename S, int L, bool ANCHOR>
__global__ void __launch_bounds__(Shape<L>::kThreads, col_blocks<S, L>())
    k_fft_cols_multi(const BatchJob *__restrict__ jobs, const uint32_t *__restrict__ col_jobs,
                     int lo, int hi, const uint32_t *__restrict__ col_units,
                     const uint16_t *__restrict__ rowbits, const uint32_t *__restrict__ counts) {
  using F = Shape<L>;
  using V = typename Vec<S>::t;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int grp = threadIdx.x / F::G, t = threadIdx.x % F::G;
  V *s = reinterpret_cast<V *>(smem_raw) + grp * F::N;
  BlockTmem<S, L> tmem(reinterpret_cast<uint32_t *>(smem_raw + col_smem_bytes<L>() - 16));
  // the block's job, in shared memory (its fields are read where used, not held
  // in registers across the transform)
  __shared__ ColJob<S> sJ;
  __shared__ uint32_t s_unit;
  for (uint32_t b = col_units[lo] + blockIdx.x; b < col_units[hi]; b += gridDim.x) {
    __syncthreads();  // the previous job's fields and buffer are no longer read
    if (threadIdx.x == 0) {
      const int k = lo + batch_job_of(col_units + lo, hi - lo, b);
      const BatchJob &B = jobs[col_jobs[k]];
      ColJob<S> &J = sJ;
      s_unit = (b - col_units[k]) * F::kGroups;
      J.cube = (const V *)B.blocked;
      J.nx = B.g.nx;
      J.ny = B.g.ny;
      J.nw = B.g.nw;
      J.w_first = B.g.w_first;
      J.nw_total = B.g.nw_total > 0 ? B.g.nw_total : B.g.nw;
      J.rowbits = rowbits + 2 * B.mask_base;
      J.counts = counts + B.counts_base;
      J.tw = (const typename fft::TwVec<S>::t *)B.tw_y;
      J.ltab = B.ltab;
      J.mtab = B.mtab;
      J.wmin = B.wmin;
      J.dw = B.dw_phase;
      J.dwnorm = B.dwnorm;
      J.norm = B.norm;
      J.phase_on = B.phase_on;
      J.anchor = B.g.nw > plain_planes<S>() ? kAnchorPlanes : B.g.nw;
      J.img_re = B.img_re;
      J.img_im = B.img_im;
      J.sums = (V *)B.cube;
    }
    __syncthreads();
    fft_col_unit<S, L, ANCHOR>(s, s_unit + grp, 0, 0, sJ.nw, false, t, sJ, tmem.addr);
  }
  tmem.release();
}

// image = norm * P * sum, P the factor of the lowest plane with data, from the sums
// of a column pass with 2^L rows: 32 columns by 64 rows a block, read along the columns
// (512 bytes a warp) and written along the rows.  FP64 sums and the image cross HBM once,
// 32 bytes a pixel (0.083 ms at 4096^2); a sincos and a root a pixel take as long, and
// 64 rows a block keep more of them in flight than 32 (523 -> 423 us for the 2048-row
// jobs of a mixed batch of 64).
constexpr int kTile = 32;
template <typename S> using FinishTile = typename Vec<S>::t[2][kTile / kLanes<S>][kTile + 1];
template <typename S, int L>
__device__ __forceinline__ void finish_tile(FinishTile<S> &tile, uint32_t n0, uint32_t m0, int low,
                                            const ColJob<S> &J) {
  constexpr int NL = kLanes<S>;
  const uint32_t lane = threadIdx.x % 32, warp = threadIdx.x / 32, warps = blockDim.x / 32;
  const uint32_t ny = (uint32_t)J.ny;
  if (low < J.nw) {
    auto at = [](uint32_t m) { return Shape<L>::kSplit ? m % 2 * Shape<L>::N + m / 2 : m; };
    const uint32_t at0 = at(m0 + lane), at1 = at(m0 + kTile + lane);
#pragma unroll 4
    for (uint32_t i = warp; i < kTile / NL; i += warps) {
      const typename Vec<S>::t *from = J.sums + (uint64_t)(n0 / NL + i) * ny;
      tile[0][i][lane] = __ldcs(from + at0);
      tile[1][i][lane] = __ldcs(from + at1);
    }
  }
  __syncthreads();
  const bool phase = J.phase_on && J.nw_total > 1;
  const double cw = __dmul_rn(2.0 * kPi, __dadd_rn(J.wmin, __dmul_rn((double)(J.w_first + low), J.dw)));
  const double l = J.ltab[n0 + lane], l2 = __dmul_rn(l, l);
#pragma unroll 1
  for (uint32_t i = warp; i < 2 * kTile; i += warps) {
    const uint32_t m = m0 + i;
    double re = 0.0, im = 0.0;
    if (low < J.nw) {
      double pr = 1.0, pi = 0.0;
      if (phase) {
        const double mm = J.mtab[m];
        const double root = __dsqrt_rn(__dsub_rn(1.0, __dadd_rn(l2, __dmul_rn(mm, mm))));
        double sn, cs;
        sincos(__dmul_rn(cw, __dsub_rn(root, 1.0)), &sn, &cs);
        const double amp = J.dwnorm * root;
        pr = cs * amp;
        pi = sn * amp;
      }
      const Cx<S> x = fft::unpack(tile[i / kTile][lane / NL][i % kTile]);
      double ar, ai;
      if constexpr (NL == 2) {
        ar = lane % 2 ? x.re.y : x.re.x;
        ai = lane % 2 ? x.im.y : x.im.x;
      } else {
        ar = x.re;
        ai = x.im;
      }
      re = J.norm * fma(ar, pr, -ai * pi);
      im = J.norm * fma(ar, pi, ai * pr);
    }
    const uint64_t o = (uint64_t)m * (uint32_t)J.nx + n0 + lane;
    __stcs(J.img_re + o, re);
    __stcs(J.img_im + o, im);
  }
}

// The lowest of a job's planes with data (nw: none), by a whole warp.
__device__ __forceinline__ int lowest_plane(const uint32_t *counts, int nw) {
  for (int w = 0; w < nw; w += 32) {
    const int k = w + (int)(threadIdx.x % 32);
    const uint32_t have = __ballot_sync(0xffffffffu, k < nw && __ldg(counts + 1 + k) > 0);
    if (have) return w + __ffs(have) - 1;
  }
  return nw;
}

constexpr int kFinishThreads = 256;

template <typename S, int L>
__global__ void __launch_bounds__(kFinishThreads) k_fft_finish(ColJob<S> J) {
  __shared__ FinishTile<S> tile;
  const uint32_t across = (uint32_t)J.nx / kTile;
  const int low = lowest_plane(J.counts, J.nw);
  finish_tile<S, L>(tile, blockIdx.x % across * kTile, blockIdx.x / across * (2 * kTile), low, J);
}

// Of the jobs col_jobs[lo..hi-1] of a batch: a block's worth of units holds
// `per_block` tiles.
template <typename S, int L>
__global__ void __launch_bounds__(kFinishThreads)
    k_fft_finish_multi(const BatchJob *__restrict__ jobs, const uint32_t *__restrict__ col_jobs, int lo,
                       int hi, const uint32_t *__restrict__ col_units, const uint32_t *__restrict__ counts) {
  constexpr uint32_t per_block = kLanes<S> * Shape<L>::kGroups * (1u << L) / (2 * kTile * kTile);
  __shared__ FinishTile<S> tile;
  const uint32_t b = col_units[lo] + blockIdx.x / per_block;
  const int k = lo + batch_job_of(col_units + lo, hi - lo, b);
  const BatchJob &B = jobs[col_jobs[k]];
  ColJob<S> J;
  J.nx = B.g.nx;
  J.ny = B.g.ny;
  J.nw = B.g.nw;
  J.w_first = B.g.w_first;
  J.nw_total = B.g.nw_total > 0 ? B.g.nw_total : B.g.nw;
  J.ltab = B.ltab;
  J.mtab = B.mtab;
  J.wmin = B.wmin;
  J.dw = B.dw_phase;
  J.dwnorm = B.dwnorm;
  J.norm = B.norm;
  J.phase_on = B.phase_on;
  J.img_re = B.img_re;
  J.img_im = B.img_im;
  J.sums = (typename Vec<S>::t *)B.cube;
  const uint32_t i = blockIdx.x - (col_units[k] - col_units[lo]) * per_block;
  const uint32_t across = (uint32_t)J.nx / kTile;
  finish_tile<S, L>(tile, i % across * kTile, i / across * (2 * kTile),
                    lowest_plane(counts + B.counts_base, J.nw), J);
}

// ---- Lists -------------------------------------------------------------------------
// Compacts the row masks of every job into its list of touched (plane, row)
// ids and per-plane counts: counts[0] = rows, counts[1 + w] = touched rows of
// plane w (at the job's counts_base).  The mask itself is turned for the column
// pass: bit r of 16-bit entry t of a plane is row t + G r (G = ny / 16; for
// ny = 8192 the halves of the plane apart, G = 256), what thread t loads.  Clears
// the image (clear_n pixels) for a column pass that adds to it.  A plan's job comes
// as a parameter (jobs null).
__global__ void k_row_list(const BatchJob *__restrict__ jobs, const __grid_constant__ BatchJob one,
                           int njobs, const uint64_t *__restrict__ mask_base, uint64_t nwords,
                           const uint32_t *__restrict__ rowmask, uint32_t *__restrict__ rowlist,
                           uint32_t *__restrict__ counts, uint16_t *__restrict__ rowbits,
                           double *__restrict__ clear_re, double *__restrict__ clear_im,
                           uint64_t clear_n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < clear_n;
       i += gridDim.x * (uint64_t)blockDim.x)
    clear_re[i] = clear_im[i] = 0.0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nwords;
       i += gridDim.x * (uint64_t)blockDim.x) {
    uint32_t bits = rowmask[i];
    const BatchJob &J = jobs ? jobs[batch_job_of(mask_base, njobs, i)] : one;
    const uint64_t li = i - J.mask_base;
    const uint32_t nty = (uint32_t)J.g.nty, ny = (uint32_t)J.g.ny;
    const uint32_t w = (uint32_t)(li / nty), band = (uint32_t)(li % nty);
    const uint32_t *plane = rowmask + J.mask_base + (uint64_t)w * nty;
    const uint32_t g = ny == 8192 ? 256 : ny / 16;
#pragma unroll
    for (uint32_t e = 2 * band; e < 2 * band + 2; e++) {
      const uint32_t k0 = e / g * (16 * g) + e % g;
      uint32_t v = 0;
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        const uint32_t k = k0 + r * g;
        v |= ((__ldg(plane + (k >> 5)) >> (k & 31)) & 1u) << r;
      }
      rowbits[2 * J.mask_base + (uint64_t)w * (ny / 16) + e] = (uint16_t)v;
    }
    if (!bits) continue;
    const uint32_t c = __popc(bits);
    uint32_t slot = atomicAdd(&counts[J.counts_base], c);
    atomicAdd(&counts[J.counts_base + 1 + w], c);
    while (bits) {
      const int b = __ffs(bits) - 1;
      bits &= bits - 1;
      const uint32_t k = band * 32 + b;
      if (k < ny) rowlist[J.list_base + slot] = w * ny + k;
      slot++;
    }
  }
}

// Row-pass units per job (blocks' worths of touched rows of its x length, `lanes`
// rows to a group), exclusive prefix over the jobs, by one warp (one thread took
// 26 us for 64 jobs; 4.5).
__global__ void k_fft_units(const BatchJob *__restrict__ jobs, int njobs, int lanes,
                            const uint32_t *__restrict__ counts, uint32_t *__restrict__ fft_units) {
  uint32_t acc = 0;
  for (int j0 = 0; j0 < njobs; j0 += 32) {
    const int j = j0 + (int)threadIdx.x;
    uint32_t n = 0;
    if (j < njobs) {
      const uint32_t rpb = (uint32_t)(fft_groups_per_block(jobs[j].logx) * lanes);
      n = (counts[jobs[j].counts_base] + rpb - 1) / rpb;
    }
    uint32_t upto = n;  // inclusive over the warp
    for (int d = 1; d < 32; d *= 2) {
      const uint32_t below = __shfl_up_sync(0xffffffffu, upto, d);
      if ((int)threadIdx.x >= d) upto += below;
    }
    if (j < njobs) fft_units[j] = acc + upto - n;
    acc += __shfl_sync(0xffffffffu, upto, 31);
  }
  if (threadIdx.x == 0) fft_units[njobs] = acc;
}

// Longest transform of the multi-job (batch) kernels: 4096.
constexpr int kMultiMaxLog = 12;

template <typename S> ColJob<S> col_job(const BatchJob &B, const FftJobs &f) {
  ColJob<S> J;
  J.cube = (const typename Vec<S>::t *)B.blocked;
  J.nx = B.g.nx;
  J.ny = B.g.ny;
  J.nw = B.g.nw;
  J.w_first = B.g.w_first;
  J.nw_total = B.g.nw_total > 0 ? B.g.nw_total : B.g.nw;
  J.rowbits = f.rowbits + 2 * B.mask_base;
  J.counts = f.counts + B.counts_base;
  J.tw = (const typename fft::TwVec<S>::t *)B.tw_y;
  J.ltab = B.ltab;
  J.mtab = B.mtab;
  J.wmin = B.wmin;
  J.dw = B.dw_phase;
  J.dwnorm = B.dwnorm;
  J.norm = B.norm;
  J.phase_on = B.phase_on;
  J.anchor = 0;  // (a plan's factors: one product over all planes)
  J.img_re = B.img_re;
  J.img_im = B.img_im;
  J.sums = (typename Vec<S>::t *)B.cube;
  return J;
}

template <typename S, int L>
int launch_rows(const FftJobs &f, const FftClass &c, cudaStream_t st) {
  using F = Shape<L>;
  using V = typename Vec<S>::t;
  constexpr int BT = F::kThreads;
  constexpr size_t sm = (size_t)BT * kVpt * 16;
  int per_sm = 0;
  if (f.one) {
    const BatchJob &B = *f.one;
    RICK_CUDA(cudaFuncSetAttribute(k_fft_rows<S, L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sm));
    RICK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fft_rows<S, L>, BT, sm));
    RICK_LAUNCHED();
    k_fft_rows<S, L><<<num_sms() * std::max(per_sm, 1), BT, sm, st>>>(
        (const typename CubeVec<S>::t *)B.cube, (V *)B.blocked, B.g.nx, B.g.ny, B.g.nty,
        (B.g.ntx + 31) / 32, f.tilemask + B.tile_base, f.rowlist + B.list_base,
        f.counts + B.counts_base, (const typename fft::TwVec<S>::t *)B.tw_x);
  } else if constexpr (L > kMultiMaxLog) {
    return set_error(RICK_ERR_INVALID_ARG, "batch FFT length above %d", 1 << kMultiMaxLog);
  } else {
    RICK_CUDA(cudaFuncSetAttribute(k_fft_rows_multi<S, L>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    RICK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fft_rows_multi<S, L>, BT, sm));
    RICK_LAUNCHED();
    k_fft_rows_multi<S, L><<<num_sms() * std::max(per_sm, 1), BT, sm, st>>>(
        f.jobs, c.lo, c.hi, f.fft_units, f.tilemask, f.rowlist, f.counts);
  }
  RICK_CUDA(cudaGetLastError());
  return RICK_OK;
}

// The column pass of one job, or of the jobs of a batch class.  The dynamic
// shared memory is padded so that shared memory, not the TMEM allocation, bounds
// the blocks per SM: a further block could not allocate and would wait for one
// of the others to finish.
template <typename S, int L>
int launch_cols(const FftJobs &f, const FftClass &c, cudaStream_t st) {
  using F = Shape<L>;
  constexpr int BT = F::kThreads, max_blocks = col_blocks<S, L>();
  if (!f.one && L > kMultiMaxLog)
    return set_error(RICK_ERR_INVALID_ARG, "batch FFT length above %d", 1 << kMultiMaxLog);
  int dev = 0, smem_sm = 0, reserved = 0;
  RICK_CUDA(cudaGetDevice(&dev));
  RICK_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  RICK_CUDA(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
  size_t sm = col_smem_bytes<L>();
  const size_t floor_b = (size_t)smem_sm / (size_t)(max_blocks + 1) + 1;
  if (sm + (size_t)reserved < floor_b) sm = floor_b - (size_t)reserved;
  sm = (sm + 15) & ~(size_t)15;
  const bool anchor = f.anchored && c.planes > plain_planes<S>() && kAnchored<S, L>;
  const void *fn = (const void *)k_fft_cols<S, L>;
  if constexpr (L <= kMultiMaxLog) {
    if (!f.one) fn = (const void *)k_fft_cols_multi<S, L, false>;
    if constexpr (kAnchored<S, L>) {
      if (!f.one && anchor) fn = (const void *)k_fft_cols_multi<S, L, true>;
    }
  }
  RICK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  // a shared-memory carveout just large enough for those blocks: the rest of the
  // SM's 256 KB stays L1, which holds the twiddles
  const int pct = (int)std::min<size_t>(
      100, ((size_t)max_blocks * (sm + (size_t)reserved) * 100 + (size_t)smem_sm - 1) / (size_t)smem_sm);
  RICK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
  const uint64_t slots = (uint64_t)num_sms() * max_blocks;
  RICK_LAUNCHED();
  if (f.one) {
    const BatchJob &B = *f.one;
    const uint64_t nb = (uint64_t)B.g.nx / kLanes<S> / F::kGroups * (F::kSplit ? 2 : 1);
    const int parts = f.cols_parts;
    const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(nb * parts, slots));
    const ColJob<S> J = col_job<S>(B, f);
    k_fft_cols<S, L><<<blocks, BT, sm, st>>>(J, parts);
    if constexpr (kFinish<L>) {
      if (parts == 1) {
        RICK_LAUNCHED();
        const uint64_t tiles = (uint64_t)J.nx * J.ny / (2 * kTile * kTile);
        k_fft_finish<S, L><<<(unsigned)tiles, kFinishThreads, 0, st>>>(J);
      }
    }
  } else if constexpr (L <= kMultiMaxLog) {
    const int blocks = (int)std::max<uint64_t>(1, std::min<uint64_t>(c.units, slots));
    if (anchor) {
      if constexpr (kAnchored<S, L>)
        k_fft_cols_multi<S, L, true><<<blocks, BT, sm, st>>>(f.jobs, f.col_jobs, c.lo, c.hi,
                                                             f.col_units, f.rowbits, f.counts);
    } else {
      k_fft_cols_multi<S, L, false><<<blocks, BT, sm, st>>>(f.jobs, f.col_jobs, c.lo, c.hi,
                                                            f.col_units, f.rowbits, f.counts);
    }
    if constexpr (kFinish<L>) {
      RICK_LAUNCHED();
      const uint64_t tiles = c.units * (uint64_t)(kLanes<S> * F::kGroups * (1 << L) / (2 * kTile * kTile));
      k_fft_finish_multi<S, L><<<(unsigned)tiles, kFinishThreads, 0, st>>>(
          f.jobs, f.col_jobs, c.lo, c.hi, f.col_units, f.counts);
    }
  }
  RICK_CUDA(cudaGetLastError());
  return RICK_OK;
}

}  // namespace

bool sparse_fft_supported(int nx, int ny) {
  // power-of-two axes from 64 to 8192 (nx >= 64 makes it a multiple of the tile)
  auto ok = [](int n) { return n >= 64 && n <= 8192 && (n & (n - 1)) == 0; };
  return ok(nx) && ok(ny);
}

// Twiddle bases of the passes (fft_core.cuh) of a transform of N = 2^L points:
// entries [0, 16) exp(2 pi i k0 / 256) of the middle pass, then
// exp(2 pi i c / N), c < N / RL, of the last one.  For 8192 points the tables of
// the even outputs (those of N = 4096) and of the odd ones (half a step on).  An
// FP32 entry carries the base's powers 1, 2, 4, 8.  Long double, rounded once.
namespace {
int twiddle_entries(int n) {
  const int halves = n == 8192 ? 2 : 1, N = n / halves;
  int L = 0;
  while ((1 << L) < N) L++;
  return halves * (16 + (N >> (L <= 8 ? L - 4 : L - 8)));
}
}  // namespace

size_t twiddle_bytes(int n, int precision) {
  return (size_t)twiddle_entries(n) *
         (precision == RICK_PREC_FP64 ? sizeof(double2) : sizeof(fft::Tw32));
}

void make_twiddles(int n, int precision, void *tab) {
  const long double two_pi = 6.283185307179586476925286766559005768L;
  const int halves = n == 8192 ? 2 : 1, N = n / halves, per = twiddle_entries(n) / halves;
  for (int h = 0; h < halves; h++)
    for (int i = 0; i < per; i++) {
      const long double turn = ((long double)(i < 16 ? i : i - 16) + 0.5L * h) /
                               (long double)(i < 16 ? 256 : N);
      for (int l = 0; l < (precision == RICK_PREC_FP64 ? 1 : 4); l++) {
        const long double a = two_pi * (turn * (long double)(1 << l));
        if (precision == RICK_PREC_FP64)
          ((double2 *)tab)[h * per + i] = make_double2((double)cosl(a), (double)sinl(a));
        else
          ((fft::Tw32 *)tab)[h * per + i].p[l] = make_float2((float)cosl(a), (float)sinl(a));
      }
    }
}

void fft_classes(const BatchJob *jobs, int njobs, int precision, FftJobs &f, uint32_t *col_jobs,
                 uint32_t *col_units) {
  f.n_row_cls = 0;
  for (int j = 0; j < njobs; j++) {
    if (f.n_row_cls == 0 || f.row_cls[f.n_row_cls - 1].log != jobs[j].logx)
      f.row_cls[f.n_row_cls++] = FftClass{jobs[j].logx, j, j + 1, 0, 0};
    else
      f.row_cls[f.n_row_cls - 1].hi = j + 1;
  }
  // column pass: the jobs grouped by logy (stable), units = blocks' worths of
  // columns (every axis a power of two of at least 64: no remainder)
  const uint32_t lanes = precision == RICK_PREC_FP64 ? 1 : 2;
  int n = 0;
  f.n_col_cls = 0;
  uint32_t acc = 0;
  for (int l = 6; l <= 13; l++) {
    const int lo = n;
    uint32_t units = 0;
    int planes = 0;
    for (int j = 0; j < njobs; j++) {
      if (jobs[j].logy != l) continue;
      col_jobs[n] = (uint32_t)j;
      col_units[n] = acc;
      const uint32_t u = (uint32_t)jobs[j].g.nx / lanes / (uint32_t)fft_groups_per_block(l);
      acc += u;
      units += u;
      planes = std::max(planes, jobs[j].g.nw);
      n++;
    }
    if (n > lo) f.col_cls[f.n_col_cls++] = FftClass{l, lo, n, units, planes};
  }
  col_units[n] = acc;
}

int sparse_fft_lists(const FftJobs &f, int precision, cudaStream_t st) {
  const uint64_t nwords = f.total_mask_words;
  const uint64_t clear = f.one && f.cols_parts > 1 ? (uint64_t)f.one->g.nx * f.one->g.ny : 0;
  const int blocks = (int)std::min<uint64_t>((std::max(nwords, clear / 8) + 255) / 256,
                                             (uint64_t)num_sms() * 8);
  RICK_LAUNCHED();
  k_row_list<<<std::max(blocks, 1), 256, 0, st>>>(
      f.one ? nullptr : f.jobs, f.one ? *f.one : BatchJob{}, f.njobs, f.mask_base, nwords, f.rowmask, f.rowlist, f.counts, f.rowbits,
      clear ? f.one->img_re : nullptr, clear ? f.one->img_im : nullptr, clear);
  RICK_CUDA(cudaGetLastError());
  if (!f.one) {  // one job's row pass reads its row count directly
    RICK_LAUNCHED();
    k_fft_units<<<1, 32, 0, st>>>(f.jobs, f.njobs, precision == RICK_PREC_FP64 ? 1 : 2, f.counts,
                                  f.fft_units);
    RICK_CUDA(cudaGetLastError());
  }
  return RICK_OK;
}

// Blocks the planes of one job's column pass are dealt to: a small image has fewer
// column blocks than the GPU has slots for them, and a block takes its planes one
// after another (64^2 x 17 FP64: 130 -> 82 us a job; 512^2 x 8, four parts, 37 ->
// 35 us a pass).  One block where that leaves each part too little: every part
// forms the pixels' steps and factors anew (1024^2 x 8 mixed in two parts 54 -> 58 us).
int column_parts(int precision, int nx, int ny, int nw) {
  int ly = 0;
  while ((1 << ly) < ny) ly++;
  const int lanes = precision == RICK_PREC_FP64 ? 1 : 2;
  const int threads = std::max(128, (ly == 13 ? 4096 : ny) / fft::kVpt);
  const int words = 2 * 4 * fft::kVpt * (lanes == 2 && ly <= 9 ? 2 : 1);  // TMEM columns of a thread
  const int64_t slots = (int64_t)num_sms() * (512 / (threads / 128 * words));
  const int64_t nb = (int64_t)nx / lanes / fft_groups_per_block(std::min(ly, 12)) * (ly == 13 ? 2 : 1);
  const int64_t room = slots / std::max<int64_t>(nb, 1);
  return room < 4 ? 1 : (int)std::min<int64_t>(nw, room);
}

#define RICK_FFT_SIZES(X) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13)

int sparse_fft_rows(const FftJobs &f, int precision, cudaStream_t st) {
  for (int i = 0; i < f.n_row_cls; i++) {
    const FftClass &c = f.row_cls[i];
    int r = RICK_ERR_INVALID_ARG;
    if (precision == RICK_PREC_FP64) {
      switch (c.log) {
#define X(L) case L: r = launch_rows<double, L>(f, c, st); break;
        RICK_FFT_SIZES(X)
#undef X
      }
    } else {
      switch (c.log) {
#define X(L) case L: r = launch_rows<float2, L>(f, c, st); break;
        RICK_FFT_SIZES(X)
#undef X
      }
    }
    RICK_TRY(r);
  }
  return RICK_OK;
}

int sparse_fft_cols(const FftJobs &f, int precision, cudaStream_t st) {
  for (int i = 0; i < f.n_col_cls; i++) {
    const FftClass &c = f.col_cls[i];
    int r = RICK_ERR_INVALID_ARG;
    if (precision == RICK_PREC_FP64) {
      switch (c.log) {
#define X(L) case L: r = launch_cols<double, L>(f, c, st); break;
        RICK_FFT_SIZES(X)
#undef X
      }
    } else {
      switch (c.log) {
#define X(L) case L: r = launch_cols<float2, L>(f, c, st); break;
        RICK_FFT_SIZES(X)
#undef X
      }
    }
    RICK_TRY(r);
  }
  return RICK_OK;
}

}  // namespace rick
