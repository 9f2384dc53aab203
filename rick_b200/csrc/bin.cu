// Device binning of visibility rows by (w-plane, grid tile).
//
// The reference grids every row with one thread that re-reads the row's
// nchan*npol samples for each of the (2K+1)^2 footprint cells
// (w-stacking.cu:104-206).  The per-cell sum
//     sum_{f,p} weight[p] * vis[f][p] * conv_weight
// factors as conv_weight * S with S = sum_{f,p} weight[p]*vis[f][p], so this
// pass reads each row's samples once, forms S in FP64 (each weight*vis product
// is the FP32 product the reference forms, w-stacking.cu:194-195; a sample whose
// real part is NaN is skipped, :191-192), and emits one compact record per grid
// tile the row's footprint touches.  Records are placed with an integer counting
// sort by (plane, tile), so the gridder reads only the rows of the tile it owns.
//
// Cell assignment is bit-exact with w-stacking.cu:143-149: FP64 IEEE division
// by dx / dw (or, for a power of two, the product with its inverse: the same bits)
// and truncation toward zero, written with explicit round-to-nearest intrinsics so
// that no multiply-add contraction can change a rounding.
#include <algorithm>

#include "rick_internal.h"

namespace rick {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kNoBin = 0xffffffffu;

struct RowPos {
  double pu, pv;  // pos_u, pos_v
  int gu, gv, gw;  // gw: plane within the shard
  bool keep;       // gridded here
  bool other;      // a valid row of a plane outside the shard
};

// gridding.c:149-188 with nsectors = 1 and yaxis = grid_size_y: the rows one
// rank grids are those of sector 0 plus the halo rows its neighbours share.
__device__ __forceinline__ bool in_sector0(double v, const Geometry &g) {
  const int binphi = (int)v;  // (int)(vvh*nsectors), nsectors = 1
  const double updist = __dsub_rn(__dmul_rn((double)((binphi + 1) * g.ny), g.dx), v);
  const double downdist = __dsub_rn(v, __dmul_rn((double)(binphi * g.ny), g.dx));
  bool in0 = (binphi == 0);
  if (binphi + 1 == 0 && updist < g.w_supporth && updist >= 0.0) in0 = true;
  if (binphi - 1 == 0 && downdist < g.w_supporth && binphi > 0 && downdist >= 0.0) in0 = true;
  return in0;
}

// w-stacking.cu:143-149.  Rows whose plane index falls outside the cube, or
// whose footprint bounds would wrap as unsigned in the reference
// (grid_u < -KernelLen), are dropped and counted.  With a w-plane shard, valid
// rows of the other shards' planes are skipped (counted apart).
__device__ __forceinline__ RowPos row_position(double u, double v, double w, const Geometry &g) {
  RowPos p;
  if (g.inv_dx > 0.0) {
    p.pu = __dmul_rn(u, g.inv_dx);
    p.pv = __dmul_rn(v, g.inv_dx);
  } else {
    p.pu = __ddiv_rn(u, g.dx);
    p.pv = __ddiv_rn(v, g.dx);
  }
  const double wi = g.inv_dw > 0.0 ? __dmul_rn(w, g.inv_dw) : __ddiv_rn(w, g.dw);
  p.gw = (int)wi;
  p.gu = (int)p.pu;
  p.gv = (int)p.pv;
  const int ntot = g.nw_total > 0 ? g.nw_total : g.nw;
  bool keep = p.gw >= 0 && p.gw < ntot && p.gu >= -g.half && p.gv >= -g.half;
  if (g.select_sector0) keep = keep && in_sector0(v, g);
  p.other = keep && (p.gw < g.w_first || p.gw >= g.w_first + g.nw);
  p.keep = keep && !p.other;
  p.gw -= g.w_first;
  return p;
}

// Bins of the (up to 2x2) tiles a footprint touches, kNoBin for unused slots
// (slot 0 is used if any is).
__device__ __forceinline__ void footprint_bins(const RowPos &p, const Geometry &g,
                                               uint32_t bins[4]) {
  bins[0] = bins[1] = bins[2] = bins[3] = kNoBin;
  if (!p.keep) return;
  const int jmin = max(p.gu - g.half, 0), jmax = min(p.gu + g.half, g.nx - 1);
  const int kmin = max(p.gv - g.half, 0), kmax = min(p.gv + g.half, g.ny - 1);
  if (jmin > jmax || kmin > kmax) return;  // footprint entirely off the grid
  const uint32_t tx0 = (uint32_t)jmin / kTile, ty0 = (uint32_t)kmin / kTile;
  const bool right = (uint32_t)jmax / kTile > tx0, down = (uint32_t)kmax / kTile > ty0;
  const uint32_t b = ((uint32_t)p.gw * g.nty + ty0) * g.ntx + tx0;  // bins fit 32 bits
  bins[0] = b;
  if (right) bins[1] = b + 1;
  if (down) bins[2] = b + g.ntx;
  if (right && down) bins[3] = b + g.ntx + 1;
}

// The same bins, packed to the front by a loop over the tiles, for the streaming
// sample pass: with the straight-line form the compiler keeps fewer of that pass's
// sample loads in flight (48 registers for 62: 2.94 ms for 1.75 at 5.1M rows of 256
// samples).
__device__ __forceinline__ void footprint_bins_packed(const RowPos &p, const Geometry &g,
                                                      uint32_t bins[4]) {
  bins[0] = bins[1] = bins[2] = bins[3] = kNoBin;
  if (!p.keep) return;
  const int jmin = max(p.gu - g.half, 0), jmax = min(p.gu + g.half, g.nx - 1);
  const int kmin = max(p.gv - g.half, 0), kmax = min(p.gv + g.half, g.ny - 1);
  if (jmin > jmax || kmin > kmax) return;  // footprint entirely off the grid
  const int tx0 = jmin / kTile, tx1 = jmax / kTile;
  const int ty0 = kmin / kTile, ty1 = kmax / kTile;
  int n = 0;
  for (int ty = ty0; ty <= ty1; ty++)
    for (int tx = tx0; tx <= tx1; tx++)
      bins[n++] = (uint32_t)(((uint64_t)p.gw * g.nty + ty) * g.ntx + tx);
}

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ void offset_bins(uint32_t bins[4], uint32_t bin_base) {
#pragma unroll
  for (int s = 0; s < 4; s++) bins[s] = bins[s] == kNoBin ? kNoBin : bins[s] + bin_base;
}

// Per-block cache of record counts: the warps of a block add into a
// direct-mapped shared table and the block adds the table into the global
// histogram once at its end, so the bins the uv centre shares across time
// steps take shared- instead of global-memory atomics.  A slot taken by
// another bin sends the count straight to the global histogram (counts stay
// exact either way).
constexpr int kCountCache = 2048;
struct CountCache {
  uint32_t key[kCountCache];
  uint32_t cnt[kCountCache];
};
__device__ __forceinline__ void cache_init(CountCache *c) {
  for (int i = threadIdx.x; i < kCountCache; i += blockDim.x) {
    c->key[i] = kNoBin;
    c->cnt[i] = 0;
  }
  __syncthreads();
}
__device__ __forceinline__ void cache_add(CountCache *c, uint32_t bin,
                                          uint32_t *__restrict__ bin_count) {
  const uint32_t h = (bin * 2654435761u) >> (32 - 11);  // multiplicative hash, 11 bits
  // a taken slot is read, not compare-and-swapped: the lanes of a warp that share a
  // bin would take turns at the swap, while the hardware adds their ones together
  uint32_t k = *(volatile uint32_t *)&c->key[h];
  if (k == kNoBin) k = atomicCAS(&c->key[h], kNoBin, bin);
  if (k == kNoBin || k == bin) atomicAdd(&c->cnt[h], 1u);
  else atomicAdd(&bin_count[bin], 1u);
}
__device__ __forceinline__ void cache_flush(CountCache *c, uint32_t *__restrict__ bin_count) {
  __syncthreads();
  for (int i = threadIdx.x; i < kCountCache; i += blockDim.x)
    if (c->cnt[i]) atomicAdd(&bin_count[c->key[i]], c->cnt[i]);
}

// Pass 1 over 32-row units u0..u1-1 of one job (rows 32 u .., one per lane):
// histogram of records per bin.  The coordinates of four units are read at once.
// Every lane adds its row's bins into the block's cache (the uv centre is dense:
// hot bins are counted in shared memory, not by global atomics; a warp-level match
// before the cache measured slower).  Counts rows dropped and rows of other shards.
constexpr int kCountUnits = 4;
__device__ __forceinline__ void count_units(const double *__restrict__ uu,
                                            const double *__restrict__ vv,
                                            const double *__restrict__ ww, uint64_t nrows,
                                            const Geometry &g, uint64_t u0, uint64_t u1,
                                            uint32_t bin_base, uint32_t *__restrict__ bin_count,
                                            uint32_t &dropped, uint32_t &other,
                                            CountCache *cache) {
  const unsigned lane = lane_id();
  for (uint64_t u = u0; u < u1; u += kCountUnits) {
    double x[kCountUnits], y[kCountUnits], z[kCountUnits];
#pragma unroll
    for (int k = 0; k < kCountUnits; k++) {
      const uint64_t i = (u + k) * 32 + lane;
      x[k] = y[k] = z[k] = 0.0;
      if (u + k < u1 && i < nrows) {
        x[k] = __ldg(uu + i);
        y[k] = __ldg(vv + i);
        z[k] = __ldg(ww + i);
      }
    }
#pragma unroll
    for (int k = 0; k < kCountUnits; k++) {
      const uint64_t i = (u + k) * 32 + lane;
      if (u + k >= u1 || i >= nrows) continue;
      const RowPos p = row_position(x[k], y[k], z[k], g);
      dropped += (p.keep || p.other) ? 0u : 1u;
      other += p.other ? 1u : 0u;
      uint32_t bins[4];
      footprint_bins(p, g, bins);
      offset_bins(bins, bin_base);
#pragma unroll
      for (int s = 0; s < 4; s++)
        if (bins[s] != kNoBin) cache_add(cache, bins[s], bin_count);
    }
  }
}

// Contiguous run of `total` units that warp `warp` of `nwarps` takes: neighbouring
// units share tiles (and, in a batch, the job).  The runs differ by one unit at most:
// with all but the last of one length, half of the warps of a pass with a few more units
// than warps had none (a mixed batch of 8 jobs of 30,011 rows of 192 samples: 546 us, 432
// so and with eight blocks an SM, one unit a warp).
__device__ __forceinline__ void warp_run(uint64_t total, uint64_t warp, uint64_t nwarps,
                                         uint64_t &u0, uint64_t &u1) {
  u0 = total * warp / nwarps;
  u1 = total * (warp + 1) / nwarps;
}

// A record in one 32-byte store (a sector).
__device__ __forceinline__ void store_record(RecF64 *to, const RecF64 &r) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(to), "d"(r.sre), "d"(r.sim),
               "d"(r.pu), "d"(r.pv)
               : "memory");
}

__device__ __forceinline__ void add_dropped(uint32_t dropped, uint32_t other, uint64_t *counters) {
  for (int o = 16; o; o >>= 1) {
    dropped += __shfl_xor_sync(kFull, dropped, o);
    other += __shfl_xor_sync(kFull, other, o);
  }
  if (lane_id() == 0 && dropped) atomicAdd((unsigned long long *)&counters[kCntDropped], dropped);
  if (lane_id() == 0 && other) atomicAdd((unsigned long long *)&counters[kCntOtherShard], other);
}

__global__ void __launch_bounds__(256, 4)
    k_bin_count(const double *__restrict__ uu, const double *__restrict__ vv,
                const double *__restrict__ ww, uint64_t nrows, Geometry g,
                uint32_t *__restrict__ bin_count, uint64_t *__restrict__ counters) {
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  __shared__ CountCache cache;
  cache_init(&cache);
  uint32_t dropped = 0, other = 0;
  uint64_t u0, u1;
  warp_run((nrows + 31) / 32, warp, nwarps, u0, u1);
  count_units(uu, vv, ww, nrows, g, u0, u1, 0, bin_count, dropped, other, &cache);
  cache_flush(&cache, bin_count);
  add_dropped(dropped, other, counters);
}

// The same over every job of a batch: a warp's run of 32-row units, job by job.
__global__ void __launch_bounds__(256, 4)
    k_bin_count_batch(const BatchJob *__restrict__ jobs, int njobs,
                      const uint64_t *__restrict__ row_units, uint64_t total_units,
                      uint32_t *__restrict__ bin_count, uint64_t *__restrict__ counters) {
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  __shared__ CountCache cache;
  cache_init(&cache);
  uint32_t dropped = 0, other = 0;
  uint64_t u, u1;
  warp_run(total_units, warp, nwarps, u, u1);
  if (u < u1) {
    int j = batch_job_of(row_units, njobs, u);
    while (u < u1) {
      while (row_units[j + 1] <= u) j++;
      const uint64_t first = row_units[j], end = min(u1, row_units[j + 1]);
      const BatchJob &J = jobs[j];
      count_units(J.uu, J.vv, J.ww, J.nrows, J.g, u - first, end - first, J.bin_base, bin_count,
                  dropped, other, &cache);
      u = end;
    }
  }
  cache_flush(&cache, bin_count);
  add_dropped(dropped, other, counters);
}

// N consecutive samples in one streaming load.
template <int N> struct SampleVec;
template <> struct SampleVec<4> { using t = float4; };
template <> struct SampleVec<2> { using t = float2; };
template <> struct SampleVec<1> { using t = float; };
template <int N>
__device__ __forceinline__ void load_samples(const float *__restrict__ p, float (&x)[N]) {
  const auto v = __ldcs(reinterpret_cast<const typename SampleVec<N>::t *>(p));
  if constexpr (N == 4) {
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
    x[3] = v.w;
  } else if constexpr (N == 2) {
    x[0] = v.x;
    x[1] = v.y;
  } else {
    x[0] = v;
  }
}

// One row's sums by one lane (loads of N, two loads of each array in flight): each
// weight*vis product is the FP32 product, a sample whose real part is NaN is skipped.
template <int N>
__device__ __forceinline__ void row_sums(const float *__restrict__ wrow,
                                         const float *__restrict__ re,
                                         const float *__restrict__ im, uint32_t npol, uint32_t nv,
                                         double &sre, double &sim) {
  if constexpr (N > 1) {
    // the polarisations (1, 2 or 4, sample_vector) repeat within a load: component c
    // of every load is polarisation c mod npol
    float wc[N];
#pragma unroll
    for (int c = 0; c < N; c++) wc[c] = __ldg(wrow + (c & (npol - 1)));
    auto add = [&](const float (&ar)[N], const float (&bi)[N]) {
#pragma unroll
      for (int c = 0; c < N; c++) {
        if (!isnan(ar[c])) {
          sre += (double)__fmul_rn(wc[c], ar[c]);
          sim += (double)__fmul_rn(wc[c], bi[c]);
        }
      }
    };
    const uint32_t nq = nv / N;
    uint32_t q = 0;
    float a0[N], b0[N], a1[N], b1[N];
    for (; q + 1 < nq; q += 2) {
      load_samples<N>(re + q * N, a0);
      load_samples<N>(im + q * N, b0);
      load_samples<N>(re + q * N + N, a1);
      load_samples<N>(im + q * N + N, b1);
      add(a0, b0);
      add(a1, b1);
    }
    if (q < nq) {
      load_samples<N>(re + q * N, a0);
      load_samples<N>(im + q * N, b0);
      add(a0, b0);
    }
  } else {
    for (uint32_t q = 0; q < nv; q++) {
      const float a = __ldcs(re + q);
      if (!isnan(a)) {
        const float wq = __ldg(wrow + (q % npol));
        sre += (double)__fmul_rn(wq, a);
        sim += (double)__fmul_rn(wq, __ldcs(im + q));
      }
    }
  }
}

// Pass 2, streaming: rows base..base+31 of a warp.  Each group of G lanes reduces
// one row's samples in loads of N; after G rounds every lane holds the sum of "its"
// row, and the records are scattered one row per lane with warp-combined cursor
// increments.  HBM-bound for long rows (5.1M rows of 256 samples: 10.8 GB in 1.75 ms,
// 0.96 of the measured copy rate); rows of eight loads run four lanes a row (3.8M
// rows of 32 samples: 0.29 ms, against 0.72 with a lane a row and 0.35 with eight).
template <int G, int N, bool SHARD>
__device__ __forceinline__ void scatter_rows(
    const double *__restrict__ uu, const double *__restrict__ vv, const double *__restrict__ ww,
    const float *__restrict__ weight, const float *__restrict__ vis_re,
    const float *__restrict__ vis_im, uint64_t nrows, uint32_t nchan, uint32_t npol,
    const Geometry &g, uint64_t base, uint32_t bin_base, const uint32_t *__restrict__ bin_off,
    uint32_t *__restrict__ bin_cursor, RecF64 *__restrict__ rec, uint32_t &gridded,
    uint32_t &nrec) {
  constexpr int R = 32 / G;  // rows per round
  const unsigned lane = lane_id();
  const unsigned sub = lane % G, grp = lane / G;
  const uint64_t nv = (uint64_t)nchan * npol;
  // With SHARD the rows of planes outside a w-plane shard (and rows that reach no
  // tile) are found before any sample is read, so they never stream their samples
  // (shard_schedule).  A whole-cube plan keeps nearly every row and compiles
  // without the check.
  bool need = true;
  if (SHARD) {
    const uint64_t i_own = base + lane;
    RowPos q;
    q.keep = false;
    if (i_own < nrows) q = row_position(uu[i_own], vv[i_own], ww[i_own], g);
    uint32_t qb[4];
    footprint_bins_packed(q, g, qb);
    need = qb[0] != kNoBin;
  }
  double my_re = 0.0, my_im = 0.0;
#pragma unroll 1
  for (int round = 0; round < G; round++) {
    const uint64_t i = base + (uint64_t)round * R + grp;
    double sre = 0.0, sim = 0.0;
    const bool need_i = __shfl_sync(kFull, need, round * R + grp);
    if (i < nrows && need_i) {
      const float *wrow = weight + i * npol;
      if (N > 1) {
        // the polarisations repeat within a load (sample_vector): component c of
        // every load is polarisation c % npol
        float wc[N];
#pragma unroll
        for (int c = 0; c < N; c++) wc[c] = __ldg(wrow + (c % npol));
        const float *re = vis_re + i * nv, *im = vis_im + i * nv;
        const uint64_t nq = nv / N;
#pragma unroll 2
        for (uint64_t q = sub; q < nq; q += G) {
          float ar[N], bi[N];
          load_samples<N>(re + q * N, ar);
          load_samples<N>(im + q * N, bi);
#pragma unroll
          for (int c = 0; c < N; c++) {
            if (!isnan(ar[c])) {
              sre += (double)__fmul_rn(wc[c], ar[c]);
              sim += (double)__fmul_rn(wc[c], bi[c]);
            }
          }
        }
      } else {
        for (uint64_t q = sub; q < nv; q += G) {
          const float a = __ldcs(vis_re + i * nv + q);
          if (!isnan(a)) {
            const float wq = __ldg(wrow + (q % npol));
            sre += (double)__fmul_rn(wq, a);
            sim += (double)__fmul_rn(wq, __ldcs(vis_im + i * nv + q));
          }
        }
      }
    }
#pragma unroll
    for (int o = G / 2; o; o >>= 1) {
      sre += __shfl_xor_sync(kFull, sre, o);
      sim += __shfl_xor_sync(kFull, sim, o);
    }
    // lane (round*R + grp') receives the sum of group grp' (its sub-lane 0)
    const int src = (int)(lane - round * R) * G;
    const double t_re = __shfl_sync(kFull, sre, src & 31);
    const double t_im = __shfl_sync(kFull, sim, src & 31);
    if (lane / R == (unsigned)round) {
      my_re = t_re;
      my_im = t_im;
    }
  }

  const uint64_t i = base + lane;
  RowPos p;
  p.keep = false;
  if (i < nrows) p = row_position(uu[i], vv[i], ww[i], g);
  uint32_t bins[4];
  footprint_bins_packed(p, g, bins);
  offset_bins(bins, bin_base);
  gridded += p.keep ? 1u : 0u;
  RecF64 r;
  r.sre = my_re;
  r.sim = my_im;
  r.pu = p.pu;
  r.pv = p.pv;
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const unsigned peers = __match_any_sync(kFull, bins[s]);
    const unsigned leader = __ffs(peers) - 1;
    uint32_t slot = 0;
    if (bins[s] != kNoBin && lane == leader) slot = atomicAdd(&bin_cursor[bins[s]], __popc(peers));
    slot = __shfl_sync(kFull, slot, leader);
    if (bins[s] != kNoBin) {
      slot += __popc(peers & ((1u << lane) - 1u));
      store_record(rec + ((uint64_t)bin_off[bins[s]] + slot), r);
      nrec++;
    }
  }
}

// Pass 2, a lane a row (rows of fewer than eight loads), of the jobs of a batch: the
// records' places are taken first -- the up to four adds of a row and the bins'
// offsets are all in flight while its samples are read; one after the other, behind
// the sums, they were most of the time (26M rows of 2 to 8 samples, 64 jobs: 2.1 ->
// 1.5 ms).
template <int N>
__device__ __forceinline__ void scatter_lane_rows(
    const double *__restrict__ uu, const double *__restrict__ vv, const double *__restrict__ ww,
    const float *__restrict__ weight, const float *__restrict__ vis_re,
    const float *__restrict__ vis_im, uint64_t i, bool valid, uint32_t nchan, uint32_t npol,
    const Geometry &g, uint32_t bin_base, const uint32_t *__restrict__ bin_off,
    uint32_t *__restrict__ bin_cursor, RecF64 *__restrict__ rec, uint32_t &gridded,
    uint32_t &nrec) {
  const unsigned lane = lane_id();
  RowPos p;
  p.keep = false;
  p.pu = p.pv = 0.0;
  if (valid) p = row_position(uu[i], vv[i], ww[i], g);
  uint32_t bins[4], slot[4], off[4];
  footprint_bins(p, g, bins);
  const bool need = bins[0] != kNoBin;
  offset_bins(bins, bin_base);
  gridded += p.keep ? 1u : 0u;
#pragma unroll
  for (int s = 0; s < 4; s++) {
    slot[s] = off[s] = 0;
    if (__any_sync(kFull, bins[s] != kNoBin)) {
      const unsigned peers = __match_any_sync(kFull, bins[s]);
      if (bins[s] != kNoBin) {
        if (lane == __ffs(peers) - 1) slot[s] = atomicAdd(&bin_cursor[bins[s]], __popc(peers));
        off[s] = __ldg(&bin_off[bins[s]]) + __popc(peers & ((1u << lane) - 1u));
      }
    }
  }
  RecF64 r;
  r.sre = r.sim = 0.0;
  if (need) {  // rows that reach no tile never stream their samples
    const uint32_t nv = nchan * npol;
    row_sums<N>(weight + i * npol, vis_re + i * nv, vis_im + i * nv, npol, nv, r.sre, r.sim);
  }
  r.pu = p.pu;
  r.pv = p.pv;
#pragma unroll
  for (int s = 0; s < 4; s++) {
    if (!__any_sync(kFull, bins[s] != kNoBin)) continue;
    const unsigned peers = __match_any_sync(kFull, bins[s]);
    const uint32_t first = __shfl_sync(kFull, slot[s], __ffs(peers) - 1);
    if (bins[s] != kNoBin) {
      store_record(rec + ((uint64_t)off[s] + first), r);
      nrec++;
    }
  }
}

__device__ __forceinline__ void add_scatter_counts(uint32_t gridded, uint32_t nrec,
                                                   uint64_t *counters) {
  for (int o = 16; o; o >>= 1) {
    gridded += __shfl_xor_sync(kFull, gridded, o);
    nrec += __shfl_xor_sync(kFull, nrec, o);
  }
  if (lane_id() == 0) {
    if (gridded) atomicAdd((unsigned long long *)&counters[kCntGridded], gridded);
    if (nrec) atomicAdd((unsigned long long *)&counters[kCntRecords], nrec);
  }
}

template <int G, int N, bool SHARD>
__global__ void __launch_bounds__(256)
    k_bin_scatter(const double *__restrict__ uu, const double *__restrict__ vv,
                  const double *__restrict__ ww, const float *__restrict__ weight,
                  const float *__restrict__ vis_re, const float *__restrict__ vis_im,
                  uint64_t nrows, uint32_t nchan, uint32_t npol, Geometry g,
                  const uint32_t *__restrict__ bin_off, uint32_t *__restrict__ bin_cursor,
                  RecF64 *__restrict__ rec, uint64_t *__restrict__ counters) {
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  uint32_t gridded = 0, nrec = 0;
  for (uint64_t base = warp * 32; base < nrows; base += nwarps * 32)
    scatter_rows<G, N, SHARD>(uu, vv, ww, weight, vis_re, vis_im, nrows, nchan, npol, g, base, 0,
                              bin_off, bin_cursor, rec, gridded, nrec);
  add_scatter_counts(gridded, nrec, counters);
}

// The same over the jobs of one sample-pass schedule of a batch (lanes per row
// G, N samples a load): the k-th listed job's rows are units sc_units[k] ..
// sc_units[k+1]-1 (a unit is 32 rows of one job).  A warp takes a run of units, so
// that the job lookup is paid once a run.
template <int G, int N>
__global__ void __launch_bounds__(256, 3)
    k_bin_scatter_batch(const BatchJob *__restrict__ jobs, const uint32_t *__restrict__ sc_jobs,
                        const uint64_t *__restrict__ sc_units, int lo, int hi,
                        const uint32_t *__restrict__ bin_off, uint32_t *__restrict__ bin_cursor,
                        RecF64 *__restrict__ rec, uint64_t *__restrict__ counters) {
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  uint32_t gridded = 0, nrec = 0;
  const uint64_t first = sc_units[lo];
  uint64_t u, u1;
  warp_run(sc_units[hi] - first, warp, nwarps, u, u1);
  u += first;
  u1 += first;
  if (u < u1) {
    int k = lo + batch_job_of(sc_units + lo, hi - lo, u);
    while (u < u1) {
      while (sc_units[k + 1] <= u) k++;
      const uint64_t j0 = sc_units[k], end = min(u1, sc_units[k + 1]);
      // the job's fields are read where used, not held in registers
      const BatchJob &J = jobs[sc_jobs[k]];
      for (; u < end; u++) {
        const uint64_t base = (u - j0) * 32;
        if constexpr (G == 1)
          scatter_lane_rows<N>(J.uu, J.vv, J.ww, J.weight, J.vis_re, J.vis_im, base + lane_id(),
                               base + lane_id() < J.nrows, J.nchan, J.npol, J.g, J.bin_base,
                               bin_off, bin_cursor, rec, gridded, nrec);
        else
          scatter_rows<G, N, false>(J.uu, J.vv, J.ww, J.weight, J.vis_re, J.vis_im, J.nrows,
                                    J.nchan, J.npol, J.g, base, J.bin_base, bin_off, bin_cursor,
                                    rec, gridded, nrec);
      }
    }
  }
  add_scatter_counts(gridded, nrec, counters);
}

// Pass 2, a lane a row (rows of fewer than eight loads), of one job: the records'
// places are taken block by block.  The uv centre is dense, so with places taken
// warp by warp its bins' cursors took an add from nearly every warp, one after
// another at one address (280k rows of 16 samples: 52 us; 31 here); the warps of a
// block add up in a shared table first, and the block adds each bin once -- while
// the samples are read.  A bin whose slots of the table are taken gets its places
// from the cursor directly.
constexpr int kShortThreads = 512;
constexpr int kPlaceSlots = 1024;
__device__ __forceinline__ uint32_t place_slot(uint32_t bin) {
  return (bin * 2654435761u) >> (32 - 10);
}
struct __align__(16) PlaceTable {
  uint32_t key[kPlaceSlots], cnt[kPlaceSlots], at[kPlaceSlots];
};

template <int N>
__global__ void __launch_bounds__(kShortThreads, 2)
    k_bin_scatter_short(const double *__restrict__ uu, const double *__restrict__ vv,
                        const double *__restrict__ ww, const float *__restrict__ weight,
                        const float *__restrict__ vis_re, const float *__restrict__ vis_im,
                        uint64_t nrows, uint32_t nchan, uint32_t npol, Geometry g,
                        const uint32_t *__restrict__ bin_off, uint32_t *__restrict__ bin_cursor,
                        RecF64 *__restrict__ rec, uint64_t *__restrict__ counters) {
  __shared__ PlaceTable place_table;
  PlaceTable *table = &place_table;
  const unsigned lane = lane_id();
  uint32_t gridded = 0, nrec = 0;
  for (uint64_t base = blockIdx.x * (uint64_t)kShortThreads; base < nrows;
       base += gridDim.x * (uint64_t)kShortThreads) {
    const uint64_t i = base + threadIdx.x;
    if (threadIdx.x < kPlaceSlots / 4) {
      reinterpret_cast<uint4 *>(table->key)[threadIdx.x] = make_uint4(kNoBin, kNoBin, kNoBin, kNoBin);
      reinterpret_cast<uint4 *>(table->cnt)[threadIdx.x] = make_uint4(0, 0, 0, 0);
    }
    RowPos p;
    p.keep = false;
    p.pu = p.pv = 0.0;
    if (i < nrows) p = row_position(__ldg(uu + i), __ldg(vv + i), __ldg(ww + i), g);
    uint32_t bins[4];
    footprint_bins(p, g, bins);
    const bool need = bins[0] != kNoBin;
    gridded += p.keep ? 1u : 0u;
    __syncthreads();  // the table is clear
    // Of the lanes with one bin the first adds for all.  place[s], on that lane: the
    // table slot and the rank so far (bit s of `in_table`), or the first place itself;
    // nobody waits for it before the records are written.
    uint32_t place[4], who[4], in_table = 0;
#pragma unroll
    for (int s = 0; s < 4; s++) {
      place[s] = who[s] = 0;
      if (!__any_sync(kFull, bins[s] != kNoBin)) continue;
      const unsigned peers = __match_any_sync(kFull, bins[s]);
      const unsigned leader = __ffs(peers) - 1;
      who[s] = leader | (uint32_t)__popc(peers & ((1u << lane) - 1u)) << 8;
      if (bins[s] != kNoBin && lane == leader) {
        const uint32_t n = __popc(peers);
        uint32_t h = place_slot(bins[s]);
        bool mine = false;
#pragma unroll
        for (int probe = 0; probe < 2 && !mine; probe++) {
          h ^= probe;  // the slot, then its neighbour
          uint32_t k = *(volatile uint32_t *)&table->key[h];
          if (k == kNoBin) k = atomicCAS(&table->key[h], kNoBin, bins[s]);
          mine = k == kNoBin || k == bins[s];
        }
        if (mine) {
          in_table |= 1u << s;
          place[s] = h << 16 | atomicAdd(&table->cnt[h], n);
        } else {
          place[s] = __ldg(&bin_off[bins[s]]) + atomicAdd(&bin_cursor[bins[s]], n);
        }
      }
    }
    __syncthreads();  // the block's counts are complete
#pragma unroll
    for (int k = threadIdx.x; k < kPlaceSlots; k += kShortThreads) {
      const uint32_t n = table->cnt[k];
      if (n) {
        const uint32_t bin = table->key[k];
        table->at[k] = __ldg(&bin_off[bin]) + atomicAdd(&bin_cursor[bin], n);
      }
    }
    RecF64 r;
    r.sre = r.sim = 0.0;
    if (need) {  // rows that reach no tile (other shards') never stream their samples
      const uint32_t nv = nchan * npol;
      row_sums<N>(weight + i * npol, vis_re + i * nv, vis_im + i * nv, npol, nv, r.sre, r.sim);
    }
    r.pu = p.pu;
    r.pv = p.pv;
    __syncthreads();  // the places are known
#pragma unroll
    for (int s = 0; s < 4; s++) {
      if (!__any_sync(kFull, bins[s] != kNoBin)) continue;
      const uint32_t first = __shfl_sync(kFull, place[s], who[s] & 31u);
      const uint32_t tab = __shfl_sync(kFull, in_table, who[s] & 31u) >> s & 1u;
      if (bins[s] == kNoBin) continue;
      const uint32_t at = (tab ? table->at[first >> 16] + (first & 0xffffu) : first) + (who[s] >> 8);
      store_record(rec + at, r);
      nrec++;
    }
    __syncthreads();  // the table is cleared for the next rows
  }
  add_scatter_counts(gridded, nrec, counters);
}

}  // namespace

// Pass 1 and the offsets: histogram of records per bin over all rows, bin
// offsets and work-item offsets (records are not written yet).
int bin_count_rows(const Geometry &g, uint64_t nrows, const double *uu, const double *vv,
                   const double *ww, Scratch &s, uint32_t max_chunk, cudaStream_t st) {
  const uint64_t nbins = g.nbins();
  if (nrows == 0) {
    RICK_CUDA(cudaMemsetAsync(s.item_off, 0, (nbins + 1) * sizeof(uint32_t), st));
    return RICK_OK;
  }
  // four units a warp where there are few: a block's cache costs its clearing and
  // its flush
  const uint64_t warps = ((nrows + 31) / 32 + kCountUnits - 1) / kCountUnits;
  const int blocks = (int)std::min<uint64_t>((warps + 7) / 8, (uint64_t)num_sms() * 8);
  RICK_LAUNCHED();
  k_bin_count<<<blocks, 256, 0, st>>>(uu, vv, ww, nrows, g, s.bin_count, s.counters);
  RICK_CUDA(cudaGetLastError());
  return scan_bins(s.bin_count, s.item_off, nbins, max_chunk, s.scan_tmp, st);
}

// Lanes that share one row's samples: one for rows of fewer than eight loads (a row
// spread over lanes would leave each lane a load or two and the warp waiting), four
// up to fifteen, then enough to cover the row's loads in one or two sweeps.
int lanes_per_row(uint64_t per_row) {
  if (per_row < 8) return 1;
  if (per_row < 16) return 4;
  return per_row < 32 ? 16 : 32;
}

// The same for a w-plane shard, and whether its rows of other planes are found
// before any sample is read (`skip`).  A whole-cube plan's schedules read every row;
// a shard leaves them where skipping is faster, on 1.5M rows with their planes in
// random order / in runs of 64 rows (us, the shard keeping half of the rows):
//   * 32 loads and more: 32 lanes, skipping (64 loads: 341 / 416 against 524 / 520
//     reading every row, 500 / 510 against 532 / 528 with nine tenths kept);
//   * 16 to 31: eight lanes, skipping (24 loads: 271 / 232 against 404 / 399 reading
//     every row and 408 / 387 skipping with sixteen lanes; 309 / 301 against 410 /
//     407 and 496 / 487 with nine tenths kept);
//   * half of the planes or more: 8 to 15 loads four lanes reading every row (12 loads:
//     150 / 144 against 268 / 222 skipping with eight lanes), fewer a lane a row with
//     block-wise places, which skips (4 loads, all but a tenth kept: 115 / 102 against
//     106 / 90 with places taken by warp, but 115 against 176 on tracks, whose dense
//     bins the block-wise places are for);
//   * less: up to 12 loads a lane a row, skipping (12 loads, a quarter of the rows kept:
//     128 / 109 against 222 / 164 with eight lanes; with block-wise places 111 / 103, but
//     381 against 320 for 3.8M rows of 8 loads on 8192^2, 16 of 64 planes, where tiles
//     share few rows), from 13 on eight lanes (15 loads, a third of the planes with 0.95
//     of the rows: 304 against 333 with a lane a row).
struct SampleSchedule {
  int lanes;
  bool skip;  // one lane without skip: block-wise places (k_bin_scatter_short)
};
static SampleSchedule shard_schedule(uint64_t per_row, bool under_half) {
  if (per_row >= 32) return {32, true};
  if (per_row >= 16) return {8, true};
  if (under_half) return {per_row >= 13 ? 8 : 1, true};
  return {per_row >= 8 ? 4 : 1, false};
}

// 16-byte loads where the rows start on 16 bytes and a load's polarisations repeat
// row by row; else 8-byte loads of pairs on the same terms.
int sample_vector(const float *vis_re, const float *vis_im, uint64_t nv, uint32_t npol) {
  const uintptr_t at = (uintptr_t)vis_re | (uintptr_t)vis_im;
  if (at % 16 == 0 && nv % 4 == 0 && (npol == 1 || npol == 2 || npol == 4)) return 4;
  if (at % 8 == 0 && nv % 2 == 0 && (npol == 1 || npol == 2)) return 2;
  return 1;
}

// Pass 2 over rows [0, nrows) of the arrays given (a contiguous slice of the
// rows pass 1 counted: records are placed through the shared bin cursors, so
// slices may follow one another in any order).
int bin_scatter_rows(const Geometry &g, uint64_t nrows, const double *uu, const double *vv,
                     const double *ww, const float *weight, const float *vis_re,
                     const float *vis_im, uint32_t nchan, uint32_t npol, Scratch &s,
                     cudaStream_t st) {
  if (nrows == 0) return RICK_OK;
  const uint64_t nv = (uint64_t)nchan * npol;
  const int N = sample_vector(vis_re, vis_im, nv, npol);
  const int sms = num_sms();
  const uint64_t per_row = nv / N;
  SampleSchedule sch{lanes_per_row(per_row), false};
  if (g.nw_total > 0 && g.nw != g.nw_total) sch = shard_schedule(per_row, 2 * g.nw < g.nw_total);
  const int G = sch.lanes;
  RICK_LAUNCHED();
  if (G == 1 && !sch.skip) {
    const uint64_t need = (nrows + kShortThreads - 1) / kShortThreads;
    const int blocks = (int)std::min<uint64_t>(need, (uint64_t)sms * 2);
#define RICK_SHORT(NN)                                                                          \
  if (N == NN)                                                                                  \
    k_bin_scatter_short<NN><<<blocks, kShortThreads, 0, st>>>(                                  \
        uu, vv, ww, weight, vis_re, vis_im, nrows, nchan, npol, g, s.bin_count, s.bin_cursor,   \
        s.records, s.counters);
    RICK_SHORT(4) RICK_SHORT(2) RICK_SHORT(1)
#undef RICK_SHORT
    RICK_CUDA(cudaGetLastError());
    return RICK_OK;
  }
  const int blocks = (int)std::min<uint64_t>(((nrows + 31) / 32 + 7) / 8, (uint64_t)sms * 8);
#define RICK_LONG(GG, NN, SKIP)                                                                  \
  if (G == GG && N == NN && sch.skip == SKIP)                                                    \
    k_bin_scatter<GG, NN, SKIP><<<blocks, 256, 0, st>>>(uu, vv, ww, weight, vis_re, vis_im,      \
                                                        nrows, nchan, npol, g, s.bin_count,      \
                                                        s.bin_cursor, s.records, s.counters);
#define RICK_SCHEDULES(NN)                                                             \
  RICK_LONG(4, NN, false) RICK_LONG(16, NN, false) RICK_LONG(32, NN, false)            \
  RICK_LONG(1, NN, true) RICK_LONG(8, NN, true) RICK_LONG(32, NN, true)
  RICK_SCHEDULES(4) RICK_SCHEDULES(2) RICK_SCHEDULES(1)
#undef RICK_SCHEDULES
#undef RICK_LONG
  RICK_CUDA(cudaGetLastError());
  return RICK_OK;
}

int bin_rows_batch(const BatchLaunch &b, Scratch &s, uint32_t max_chunk, cudaStream_t st) {
  const uint64_t nbins = b.total_bins;
  const int sms = num_sms();
  const uint64_t units = b.total_row_units;
  const uint64_t warps = (units + kCountUnits - 1) / kCountUnits;
  const int blocks_cnt =
      (int)std::max<uint64_t>(1, std::min<uint64_t>((warps + 7) / 8, (uint64_t)sms * 8));
  RICK_LAUNCHED();
  k_bin_count_batch<<<blocks_cnt, 256, 0, st>>>(b.jobs, b.njobs, b.u.row_units, units,
                                                s.bin_count, s.counters);
  RICK_CUDA(cudaGetLastError());
  RICK_TRY(scan_bins(s.bin_count, s.item_off, nbins, max_chunk, s.scan_tmp, st));
  for (int c = 0; c < b.n_sc; c++) {
    const ScatterClass &k = b.sc[c];
    const int blocks = (int)std::max<uint64_t>(
        1, std::min<uint64_t>((k.units + 7) / 8, (uint64_t)sms * (k.lanes > 1 ? 8 : 6)));
    RICK_LAUNCHED();
#define RICK_SC(GG, NN)                                                                      \
  if (k.lanes == GG && k.vec == NN)                                                          \
    k_bin_scatter_batch<GG, NN><<<blocks, 256, 0, st>>>(b.jobs, b.sc_jobs, b.sc_units, k.lo, \
                                                        k.hi, s.bin_count, s.bin_cursor,     \
                                                        s.records, s.counters);
#define RICK_LANES(NN) RICK_SC(1, NN) RICK_SC(4, NN) RICK_SC(16, NN) RICK_SC(32, NN)
    RICK_LANES(4) RICK_LANES(2) RICK_LANES(1)
#undef RICK_LANES
#undef RICK_SC
    RICK_CUDA(cudaGetLastError());
  }
  return RICK_OK;
}

}  // namespace rick
