// In-place power-of-two inverse FFTs in shared memory, 16 values per thread.
//
// A transform of N = 2^L points (64..4096) is run by G = N/16 threads in two or
// three passes of decimation in time: radix 16, radix 16 (N >= 512), and a last
// radix RL of 2..16.  Writing n = n0 + RL n1 + G n2 for the input index and k0,
// k1, k2 for the output digits found by the passes, element (n0, n1, k0) of a
// pass lives at n0 + RL n1 + G k0: each thread writes a pass's results where it
// read the pass's inputs, so an exchange takes one barrier (the autosorting
// order this replaces took two), and the outputs of the last pass stay in
// registers, thread t holding t + G q (q = 0..15).  Sixteen values per thread
// make two exchanges of a 4096-point transform where radix 8 made three; the
// shared-memory pipe bounds these kernels beside the FP64 pipe.
//
// Each radix-2 butterfly takes its twiddle in the same step: a + w b in four
// fused multiply-adds and a - w b as 2 a - (a + w b) in two (FP64), six
// instructions for the eight of a product and two sums.
//
// The element type S is double, or float2: the same element of two transforms
// (two image columns, two grid rows) in packed FP32 instructions (fma.f32x2),
// which issue two operations per lane.  Both take 16 bytes per complex element,
// so both forms share every index, barrier and copy.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace rick {
namespace fft {

constexpr int kVpt = 16;  // values per thread

// ---- arithmetic on S -----------------------------------------------------------
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double fma_(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double neg(double a) { return -a; }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma_(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
template <typename S> __device__ __forceinline__ S splat(double c);
template <> __device__ __forceinline__ double splat<double>(double c) { return c; }
template <> __device__ __forceinline__ float2 splat<float2>(double c) {
  return make_float2((float)c, (float)c);
}

// Transforms one element carries.
template <typename S> constexpr int kLanes = 1;
template <> constexpr int kLanes<float2> = 2;

template <typename S> struct Cx {
  S re, im;
};
template <typename S>
__device__ __forceinline__ Cx<S> cmul(Cx<S> a, Cx<S> b) {
  return {fma_(a.re, b.re, neg(mul(a.im, b.im))), fma_(a.re, b.im, mul(a.im, b.re))};
}
template <typename S>
__device__ __forceinline__ Cx<S> csquare(Cx<S> a) {
  const S t = mul(a.re, a.im);
  return {fma_(a.re, a.re, neg(mul(a.im, a.im))), add(t, t)};
}

// A value as it lies in memory: 16 bytes, re then im.
template <typename S> struct Vec;
template <> struct Vec<double> { using t = double2; };
template <> struct Vec<float2> { using t = float4; };
__device__ __forceinline__ Cx<double> unpack(double2 v) { return {v.x, v.y}; }
__device__ __forceinline__ Cx<float2> unpack(float4 v) {
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ double2 pack(Cx<double> c) { return make_double2(c.re, c.im); }
__device__ __forceinline__ float4 pack(Cx<float2> c) {
  return make_float4(c.re.x, c.re.y, c.im.x, c.im.y);
}
// The twiddle base w of a butterfly and its powers w^2, w^4, w^8.  FP64 squares
// them from the table's w; FP32 reads all four from the table (each rounded once:
// squaring would leave w^8 several ulp off, which shows in the image).
template <typename S> struct Tw {
  Cx<S> p[4];
};
template <typename S> struct TwVec;  // a table entry in memory
template <> struct TwVec<double> { using t = double2; };
struct __align__(16) Tw32 {
  float2 p[4];
};
template <> struct TwVec<float2> { using t = Tw32; };
__device__ __forceinline__ Tw<double> twiddle(const double2 *__restrict__ e) {
  const double2 v = __ldg(e);
  Tw<double> w;
  w.p[0] = {v.x, v.y};
#pragma unroll
  for (int l = 1; l < 4; l++) w.p[l] = csquare(w.p[l - 1]);
  return w;
}
__device__ __forceinline__ Tw<float2> twiddle(const Tw32 *__restrict__ e) {
  const float4 a = __ldg(reinterpret_cast<const float4 *>(e));
  const float4 b = __ldg(reinterpret_cast<const float4 *>(e) + 1);
  Tw<float2> w;
  w.p[0] = {make_float2(a.x, a.x), make_float2(a.y, a.y)};
  w.p[1] = {make_float2(a.z, a.z), make_float2(a.w, a.w)};
  w.p[2] = {make_float2(b.x, b.x), make_float2(b.y, b.y)};
  w.p[3] = {make_float2(b.z, b.z), make_float2(b.w, b.w)};
  return w;
}
// Entry ex in lane x, ey in lane y.
__device__ __forceinline__ Tw<float2> twiddle(const Tw32 *__restrict__ ex,
                                              const Tw32 *__restrict__ ey) {
  Tw<float2> w = twiddle(ex);
  const Tw<float2> y = twiddle(ey);
#pragma unroll
  for (int l = 0; l < 4; l++) {
    w.p[l].re.y = y.p[l].re.y;
    w.p[l].im.y = y.p[l].im.y;
  }
  return w;
}

// ---- butterflies ---------------------------------------------------------------
// (a, b) <- (a + w b, a - w b), and the same with i w for w.
template <typename S> __device__ __forceinline__ void bfly(Cx<S> &a, Cx<S> &b, Cx<S> w) {
  const S two = splat<S>(2.0);
  const Cx<S> p = {fma_(neg(w.im), b.im, fma_(w.re, b.re, a.re)),
                   fma_(w.im, b.re, fma_(w.re, b.im, a.im))};
  b = {fma_(two, a.re, neg(p.re)), fma_(two, a.im, neg(p.im))};
  a = p;
}
template <typename S> __device__ __forceinline__ void bfly_i(Cx<S> &a, Cx<S> &b, Cx<S> w) {
  const S two = splat<S>(2.0);
  const Cx<S> p = {fma_(neg(w.re), b.im, fma_(neg(w.im), b.re, a.re)),
                   fma_(neg(w.im), b.im, fma_(w.re, b.re, a.im))};
  b = {fma_(two, a.re, neg(p.re)), fma_(two, a.im, neg(p.im))};
  a = p;
}
template <typename S> __device__ __forceinline__ void bfly_1(Cx<S> &a, Cx<S> &b) {
  const Cx<S> p = {add(a.re, b.re), add(a.im, b.im)};
  b = {sub(a.re, b.re), sub(a.im, b.im)};
  a = p;
}
template <typename S> __device__ __forceinline__ void bfly_1i(Cx<S> &a, Cx<S> &b) {
  const Cx<S> p = {sub(a.re, b.im), add(a.im, b.re)};
  b = {add(a.re, b.im), sub(a.im, b.re)};
  a = p;
}
// w exp(+2 pi i j / 16), j = 0..3 known after unrolling.
template <typename S> __device__ __forceinline__ Cx<S> rot16(Cx<S> w, int j) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
  constexpr double h = 0.70710678118654752440;
  switch (j) {
    case 0: return w;
    case 1: return cmul(w, Cx<S>{splat<S>(c1), splat<S>(s1)});
    case 2: return {mul(sub(w.re, w.im), splat<S>(h)), mul(add(w.re, w.im), splat<S>(h))};
    default: return cmul(w, Cx<S>{splat<S>(s1), splat<S>(c1)});
  }
}
template <typename S> __device__ __forceinline__ Cx<S> const16(int j) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
  constexpr double h = 0.70710678118654752440;
  switch (j) {
    case 1: return {splat<S>(c1), splat<S>(s1)};
    case 2: return {splat<S>(h), splat<S>(h)};
    default: return {splat<S>(s1), splat<S>(c1)};
  }
}

__host__ __device__ constexpr int bitrev(int v, int bits) {
  int r = 0;
  for (int i = 0; i < bits; i++) r |= ((v >> i) & 1) << (bits - 1 - i);
  return r;
}
__host__ __device__ constexpr int ilog2(int n) { return n <= 1 ? 0 : 1 + ilog2(n / 2); }

// Inverse DFT of the R values x[r] w^r (w = 1 without TW); output k is left in
// x[bitrev(k)].  The combination of r and r + h multiplies by z^h with
// z = w exp(2 pi i k / R), which depends on k modulo R/h only: level by level
// the classes of k double, and the upper half of them is i times the lower.
template <int R, bool TW, typename S>
__device__ __forceinline__ void dft(Cx<S> *x, const Tw<S> &w) {
  constexpr int LR = ilog2(R);
#pragma unroll
  for (int lev = 0; lev < LR; lev++) {
    const int h = R >> (lev + 1), half = lev > 0 ? 1 << (lev - 1) : 1;
#pragma unroll
    for (int c = 0; c < half; c++) {
      const int j = c * h * (16 / R);  // class c turns by exp(2 pi i j / 16), j < 4
      Cx<S> z;
      if constexpr (TW) z = rot16(w.p[LR - 1 - lev], j);
      else z = const16<S>(j);
      const int base = lev > 0 ? bitrev(c, lev) * 2 * h : 0;
#pragma unroll
      for (int r = 0; r < h; r++) {
        if (TW || j != 0) bfly(x[base + r], x[base + r + h], z);
        else bfly_1(x[base + r], x[base + r + h]);
      }
      if (lev > 0) {
        const int base_i = bitrev(c + half, lev) * 2 * h;
#pragma unroll
        for (int r = 0; r < h; r++) {
          if (TW || j != 0) bfly_i(x[base_i + r], x[base_i + r + h], z);
          else bfly_1i(x[base_i + r], x[base_i + r + h]);
        }
      }
    }
  }
}

// ---- the transform of 2^L points (L = 6..12; 13: half of the outputs) -------------
// L = 13: the even or odd outputs (half c = 0 or 1) of an 8192-point transform,
// as a 4096-point one over x[n] + x[n+4096] or x[n] - x[n+4096] evaluated at
// frequencies k + c/2: every twiddle base gains half a step.
template <int L> struct Shape {
  static constexpr int kLog = L == 13 ? 12 : L;       // transform run by a group
  static constexpr bool kSplit = L == 13;
  static constexpr int N = 1 << kLog, G = N / kVpt;   // points, threads of a group
  static constexpr int kPasses = kLog <= 8 ? 2 : 3;
  static constexpr int LR = kPasses == 2 ? kLog - 4 : kLog - 8;
  static constexpr int RL = 1 << LR, B = kVpt / RL;   // last radix, its butterflies per thread
  static constexpr int kThreads = G > 128 ? G : 128;  // a block
  static constexpr int kGroups = kThreads / G;        // transforms per block
  static constexpr int kLast = 16;                    // twiddle table: [0,16) mid, then the last
  static constexpr int kTab = 16 + N / RL;            // entries of one half's table
};

// Shared-memory position of element `low` + G k0 (low < G): the low three bits
// turned by the bit-reversed k0, so that the lanes of every pass's access fall
// on distinct 16-byte banks (runs of eight consecutive `low`, of eight k0, and
// of 4 x 2 or 2 x 4 where the last radix is 4 or 2).  At N = 64 a group has four
// positions per k0: two bits.
template <int L> __device__ __forceinline__ int spos(int low, int k0) {
  using F = Shape<L>;
  const int f = F::G >= 8 ? ((k0 & 1) << 2) | (k0 & 2) | ((k0 >> 2) & 1) : (k0 & 3);
  return (low ^ f) + F::G * k0;
}

// The barrier of the threads of one group.
template <int L> __device__ __forceinline__ void group_sync() {
  using F = Shape<L>;
  if constexpr (F::G <= 32) {
    __syncwarp();
  } else if constexpr (F::kGroups == 1) {
    __syncthreads();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / F::G), "n"(F::G) : "memory");
  }
}

// What the element type's lanes of a 13-bit transform hold: one half of the
// outputs, or (float2 only) the even outputs in lane x and the odd ones in y.
enum Half { kEven = 0, kOdd = 1, kBoth = 2 };

// exp(2 pi i / 32) and its powers: the first pass of an 8192-point transform's odd
// outputs.
template <typename S> __device__ __forceinline__ Tw<S> odd_base() {
  constexpr double c32 = 0.98078528040323044913, s32 = 0.19509032201612826785;
  Tw<S> w;
  w.p[0] = {splat<S>(c32), splat<S>(s32)};
  w.p[1] = const16<S>(1);
  w.p[2] = const16<S>(2);
  w.p[3] = {splat<S>(0.0), splat<S>(1.0)};
  return w;
}

// First pass of the group's thread t: v[r] is input t + G r.  Leaves the values
// in shared memory, behind a barrier that frees the buffer (every thread has read
// its previous contents) -- placed after the arithmetic, where it costs least.
template <int L, typename S>
__device__ __forceinline__ void first_pass(typename Vec<S>::t *s, int t, int half,
                                           Cx<S> (&v)[kVpt]) {
  using F = Shape<L>;
  if constexpr (F::kSplit) {
    if (half == kOdd) {
      dft<16, true, S>(v, odd_base<S>());
    } else if (half == kBoth) {
      Tw<S> w = odd_base<S>();
      if constexpr (kLanes<S> == 2) {
#pragma unroll
        for (int l = 0; l < 4; l++) {
          w.p[l].re.x = 1.0f;
          w.p[l].im.x = 0.0f;
        }
      }
      dft<16, true, S>(v, w);
    } else {
      dft<16, false, S>(v, Tw<S>{});
    }
  } else {
    dft<16, false, S>(v, Tw<S>{});
  }
  group_sync<L>();
#pragma unroll
  for (int r = 0; r < 16; r++) s[spos<L>(t, r)] = pack(v[bitrev(r, 4)]);
}

// The passes after the first: v[q] becomes output t + G q.  The caller has not
// passed the barrier after the first pass's stores yet: each pass's
// twiddle is read ahead of the barrier before it, while no values are held.
// tw(e): entry e of the transform's twiddle table as an element ([0, 16) the
// middle pass, kLast.. the last one).
template <int L, typename S, typename TwOf>
__device__ __forceinline__ void later_passes(typename Vec<S>::t *s, int t, TwOf tw,
                                             Cx<S> (&v)[kVpt]) {
  using F = Shape<L>;
  constexpr int RL = F::RL, G = F::G;
  if constexpr (F::kPasses == 3) {
    const int n0 = t % RL, k0 = t / RL;
    const Tw<S> w = tw(k0);
    group_sync<L>();
#pragma unroll
    for (int r = 0; r < 16; r++) v[r] = unpack(s[spos<L>(n0 + RL * r, k0)]);
    dft<16, true, S>(v, w);
#pragma unroll
    for (int r = 0; r < 16; r++) s[spos<L>(n0 + RL * r, k0)] = pack(v[bitrev(r, 4)]);
  }
  Tw<S> w[F::B];
  Cx<S> x[kVpt];
#pragma unroll
  for (int j = 0; j < F::B; j++) w[j] = tw(F::kLast + t + G * j);
  group_sync<L>();
#pragma unroll
  for (int j = 0; j < F::B; j++) {
    const int c = t + G * j;
    const int k0 = F::kPasses == 3 ? t & 15 : c, k1 = F::kPasses == 3 ? c >> 4 : 0;
#pragma unroll
    for (int r = 0; r < RL; r++) x[j * RL + r] = unpack(s[spos<L>(RL * k1 + r, k0)]);
  }
#pragma unroll
  for (int j = 0; j < F::B; j++) {
    dft<RL, true, S>(x + j * RL, w[j]);
#pragma unroll
    for (int k = 0; k < RL; k++) v[j + F::B * k] = x[j * RL + bitrev(k, F::LR)];
  }
}

}  // namespace fft
}  // namespace rick
