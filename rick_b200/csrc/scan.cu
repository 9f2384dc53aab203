// Offsets of the bins and of the gridder's work items: exclusive prefix sums of the
// record counts and of ceil(count / max_chunk), both at once.  One block for up to
// 8191 bins; beyond, a first kernel sums blocks of 8192 bins and a second adds the
// sums before its block (read by every block: 512 at 4M bins) to the
// block's own scan.  The scans of one sum at a time this replaces took seven
// launches for 8,192 bins.
#include "rick_internal.h"

namespace rick {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanPerThread = 8;
constexpr int kScanBlock = kScanThreads * kScanPerThread;

// Records and work items, summed together.
struct Sum2 {
  uint32_t rec, items;
};
__device__ __forceinline__ Sum2 operator+(Sum2 a, Sum2 b) {
  return {a.rec + b.rec, a.items + b.items};
}

__device__ __forceinline__ Sum2 warp_inclusive(Sum2 v) {
  const unsigned lane = threadIdx.x & 31u;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Sum2 t = {__shfl_up_sync(0xffffffffu, v.rec, o), __shfl_up_sync(0xffffffffu, v.items, o)};
    if (lane >= (unsigned)o) v = v + t;
  }
  return v;
}

// Exclusive prefix of each thread's value over the block, and the block's total.
__device__ __forceinline__ Sum2 block_exclusive(Sum2 v, Sum2 &total) {
  __shared__ Sum2 warp_tot[kScanThreads / 32];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const Sum2 incl = warp_inclusive(v);
  __syncthreads();  // warp_tot of an earlier call is no longer read
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  const Sum2 t = warp_inclusive(warp_tot[lane]);  // every warp scans the warps' totals
  total = {__shfl_sync(0xffffffffu, t.rec, 31), __shfl_sync(0xffffffffu, t.items, 31)};
  const int src = warp == 0 ? 0 : (int)warp - 1;
  const Sum2 before = {__shfl_sync(0xffffffffu, t.rec, src), __shfl_sync(0xffffffffu, t.items, src)};
  const Sum2 own = {incl.rec - v.rec, incl.items - v.items};
  return warp == 0 ? own : own + before;
}

__device__ __forceinline__ Sum2 bin_sum(uint32_t c, uint32_t max_chunk) {
  return {c, (c + max_chunk - 1) / max_chunk};
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_sums(const uint32_t *__restrict__ counts, uint64_t nbins, uint32_t max_chunk,
                Sum2 *__restrict__ sums) {
  const uint64_t base = (uint64_t)blockIdx.x * kScanBlock + threadIdx.x;
  Sum2 local = {0, 0}, total;
#pragma unroll
  for (int k = 0; k < kScanPerThread; k++) {
    const uint64_t i = base + (uint64_t)k * kScanThreads;
    if (i < nbins) local = local + bin_sum(counts[i], max_chunk);
  }
  block_exclusive(local, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// sums: the totals of the blocks (null for a single block).
__global__ void __launch_bounds__(kScanThreads)
    k_scan_bins(uint32_t *__restrict__ counts, uint32_t *__restrict__ item_off, uint64_t nbins,
                uint32_t max_chunk, const Sum2 *__restrict__ sums) {
  Sum2 before = {0, 0}, total;
  if (sums) {
    Sum2 part = {0, 0};
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kScanThreads) part = part + sums[b];
    block_exclusive(part, before);
  }
  const uint64_t base = (uint64_t)blockIdx.x * kScanBlock + (uint64_t)threadIdx.x * kScanPerThread;
  Sum2 v[kScanPerThread], local = {0, 0};
#pragma unroll
  for (int k = 0; k < kScanPerThread; k++) {
    v[k] = bin_sum(base + k < nbins ? counts[base + k] : 0u, max_chunk);
    local = local + v[k];
  }
  Sum2 run = before + block_exclusive(local, total);
#pragma unroll
  for (int k = 0; k < kScanPerThread; k++) {
    if (base + k <= nbins) {  // entry nbins: the totals
      counts[base + k] = run.rec;
      item_off[base + k] = run.items;
    }
    run = run + v[k];
  }
}

}  // namespace

// Two words a block of 8192 bins, with room to spare.
uint64_t scan_tmp_words(uint64_t n) {
  uint64_t words = 0;
  while (n > 4096) {
    n = (n + 4095) / 4096;
    words += n;
  }
  return words + 64;
}

int scan_bins(uint32_t *counts, uint32_t *item_off, uint64_t nbins, uint32_t max_chunk,
              uint32_t *tmp, cudaStream_t st) {
  const uint64_t nb = (nbins + 1 + kScanBlock - 1) / kScanBlock;
  Sum2 *sums = nb > 1 ? (Sum2 *)tmp : nullptr;
  if (sums) {
    RICK_LAUNCHED();
    k_scan_sums<<<(unsigned)nb, kScanThreads, 0, st>>>(counts, nbins, max_chunk, sums);
    RICK_CUDA(cudaGetLastError());
  }
  RICK_LAUNCHED();
  k_scan_bins<<<(unsigned)nb, kScanThreads, 0, st>>>(counts, item_off, nbins, max_chunk, sums);
  RICK_CUDA(cudaGetLastError());
  return RICK_OK;
}

}  // namespace rick
