// IHC + lambda with the AC filter on the tensor cores: the same stage as
// ihc_lambda.cu's kernel, bit for bit, for filters of up to 257 taps.
//
// What bounded the stage: 127 tap pairs of compensated FP32 arithmetic per
// point, ~2,170 lane operations (43 ms of the FP32 pipe on 2.9 million rows).
// Here the filter is a product of digit matrices (tensor_fir.cuh) that is exact
// to about 2^-50 of the scales, 23k cycles of the tensor pipe for a tile of
// 128 rows x 64 sections; six exact integers per point leave TMEM.
//
// The same bits as the compensated FIR (Dot2).  Both are the sum rounded once,
// up to errors far below an ulp: the digits', and Dot2's, over 400,000 points of
// solved velocity (tones of 20-100 dB, noise of 0-40 dB) at most 59 x 2^-48 of
// the largest partial sum among four rows of a tile.  So the two can only differ
// where the exact sum lies that close to a rounding boundary.  The tile bounds its
// first and last row's partial sums from above (sums from either end of the
// filter over runs of 24 rows, from registers); the epilogue rounds the sum +-
// 40 x 2^-48 of that bound, about twice the partial sum itself; where it makes a
// difference, and in rows whose look-back is shorter than the tile's, the point
// is evaluated by Dot2.  On the JND sweep 39% of the tiles have no such point,
// 48% one to eight of 8,192.  (The 59 is measured, not proven: a point past it would be
// the exact sum's rounding where Dot2's is the other neighbour of a tie.)
//
// Not below a floor, which bounds the error of the digits' sum (ihc_tensor_taps): what the
// digits leave of x and of the taps, and the pairs left out.  It decides where a section's
// sums are tiny beside its largest |x|, as at the start of a segment, whose velocity grows
// from nothing by orders of magnitude within a tile.  (Five digits of x, and six standard
// deviations of what they leave: steady values of 2^-22 of the tile's largest came out as
// the other neighbour.  Five digits and the bound of what they leave: 33 intervals
// 1.41 -> 1.54 ms, with the remainders' own maximum 1.50; six digits 1.43.)
//
// Some inputs leave nearly all points in doubt for long: tones in a null of the filter (a
// sum 2^-20 of its partial sums), a stop band of 100 dB, values below the digits' range.
// A tile of 128 rows then costs what it costs on the FP32 pipe, and the products' part in
// vain: such tiles are told from the start of a segment by their last rows, and after two
// of them the next are taken without products, eight rows to a warp (ac_blocks), while
// half of the warps finish the tile before.  100,000 rows of a 2 kHz tone, which the 255
// taps have a null at: row by row 4.25 ms, so 2.63 (FP32 kernel 2.41); a Blackman window,
// 4 kHz 4.18 -> 2.61 (2.39); 60,000 rows below 2^-80 2.90 -> 1.73 (1.60).  At once after
// the first such tile: 2.60 and 0.90 instead of 0.86 for 125 Hz; none finished before the
// next is begun: 2.73 and 0.84.
//
// One CTA: 64 sections x a run of tiles of one frame.  Sixteen warps hold the
// tile's 384 rows of velocity in registers (48 values a thread) and write one
// digit after another into two shared-memory halves; a seventeenth issues the
// products as soon as a half is there.  Between the digits the same warps finish
// the tile before: its Dot2 points, the DC sums, IHC and lambda.
//
// What bounds it now: the workers' chain, ~54k cycles a tile (Dot2 points 7k, DC
// sums 11k, IHC / lambda 7k, loads 7k, digits 12k, epilogue 4k) at 41% of the
// issue slots, not the tensor pipe.  Finishing a tile at once instead of between
// the next one's digits takes 22.0 ms against 18.9 (JND sweep); without the products
// (accumulators left as they are) the chain takes the same time.  Single points by
// a warp whose lanes share the work (sym_point): 18.65 -> 17.5 ms.  DC sums whose
// errors run a batch behind, or on two blocks at once: 19.5 and 19.6 against 18.65.
// Where there are too many points for the list, a bit each says which, instead of all
// rows of the tile: one signal 304 -> 262 us, 33 intervals 1.46 -> 1.44 ms.
//
// Measured (GB300), against the FP32 pipe: JND sweep (2.9 million rows) 53.7 ->
// 18.0 ms, 176,000 rows in 33 intervals 4.46 -> 1.43 ms, one signal of 5,330 rows
// 0.80 -> 0.26 ms.

#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
#include <limits>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "ihc_common.cuh"
#include "ihc_tensor.h"
#include "tensor_fir.cuh"

namespace cgb {
namespace {

constexpr int kWorkers = kIhcWarps * 32;   // threads that do everything but issue
constexpr int kThreads = kWorkers + 128;   // the issuing warp's group of four
// registers a thread: 96 at launch (640 threads), then 112 for the workers and
// 32 for the issuing warp's group, together the same
constexpr int kWorkerRegs = 112, kIssueRegs = 32;
static_assert(kWorkers * kWorkerRegs + 128 * kIssueRegs <= kThreads * 96, "register split");
constexpr int kCols = tfir::kCols;
constexpr int kPitch = kCols + 1;          // a row of dS / AC: lanes along rows too
constexpr int kGroups = kCols / 32;        // section halves
constexpr int kList = 1024;                // points for Dot2 listed by tile
constexpr int kFewPoints = 48;             // up to here a warp to a point
constexpr int kLate = 256;                 // of the last 32 rows, from which more will follow
constexpr int kDirectTiles = 15;           // tiles without products before they are tried again
constexpr int kRuns = 16;                  // runs of 24 rows of a tile's x

// A warp's scratch for one point (sym_point).
constexpr int kPairs = tfir::kMaxTaps / 2;
struct __align__(16) PointScratch {
  float p[kPairs];   // products; then the running sums; then the errors
  float ep[kPairs];  // errors of the pairs' sums
};

struct TensorShared {
  uint64_t mbar[2];          // products of half h are done
  uint64_t ready[2];         // a digit of half h is in shared memory (a warp, an arrival)
  uint64_t drained;          // all products that were issued are done
  uint32_t tmem;
  int abort;                 // a wait ran out
  int stop;                  // the workers have issued their last digit
  int listed;                // points for Dot2 (more than kList: those flagged)
  int late;                  // those in the tile's last 32 rows
  int dot2_rows[2];          // rows for Dot2, by tile parity
  int kmin[2];               // first row of x of the tile, by tile parity
  uint32_t top[2][kCols];    // largest |x| bits of the tile, by tile parity
  alignas(16) float2 scale[kCols];       // slack in units of the accumulators (+inf: no usable
                             // scale), and the unit 2^(e+eb-16)
  uint32_t partial[kCols];   // bits of the largest partial sum of the sampled rows
  // of the first and last row's sum over each run of 24 rows of x: the sum and
  // its largest partial sum
  // (each warp's scratch when single points are evaluated, after their use)
  union {
    alignas(16) float2 sample[2][kRuns][kCols];
    PointScratch point[kIhcWarps];
  };
  uint16_t list[kList];
  alignas(4) unsigned char flag[tfir::kRows][kCols / 8];  // the points for Dot2, a bit each
  unsigned char row[tfir::kRows];  // how the tile's row gets its AC: kRow...
};
static_assert(offsetof(TensorShared, mbar) % 8 == 0 && offsetof(TensorShared, scale) % 16 == 0 &&
                  offsetof(TensorShared, sample) % 8 == 0 && sizeof(TensorShared) % 16 == 0,
              "vector accesses");
constexpr int kRowZero = 0, kRowSum = 1, kRowDot2 = 2;

__device__ __forceinline__ void sync_workers() {
  asm volatile("bar.sync 3, %0;" ::"n"(kWorkers) : "memory");
}
// Workers: this warp's share of half h of a digit is in shared memory.
__device__ __forceinline__ void half_ready(TensorShared& S, int h, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(&S.ready[h]);
}
// The issuing warp, converged: phase `n` of ready[h]; false where there is none, or a
// wait of the workers, or this one, ran out.
__device__ __forceinline__ bool half_wait(TensorShared& S, int h, int n) {
  const unsigned long long start = global_ns();
  while (!__all_sync(kFull, mbar_done(&S.ready[h], n))) {
    // (the workers' steps between two digits are far shorter, their waits a fourth)
    const bool late = global_ns() - start > 4 * kWaitNs;
    if (__any_sync(kFull, late || *(volatile int*)&S.abort || *(volatile int*)&S.stop))
      return false;
  }
  return true;
}

// TwoSum, two at once
__device__ __forceinline__ float2 two_sum2(float2 a, float2 b, float2& err) {
  const float2 t = add2(a, b);
  const float2 z = sub2(t, a);
  err = add2(sub2(a, sub2(t, z)), sub2(b, z));
  return t;
}

// own_log10f on a pair: the same operation sequence per element.
__device__ __forceinline__ float2 own_log10f2(float2 x) {
  const int ix = __float_as_int(x.x), iy = __float_as_int(x.y);
  float mx = __int_as_float((ix & 0x7fffff) | 0x3f800000);
  float my = __int_as_float((iy & 0x7fffff) | 0x3f800000);
  const bool hx = mx > 1.41421356f, hy = my > 1.41421356f;
  mx = hx ? __fmul_rn(mx, 0.5f) : mx;
  my = hy ? __fmul_rn(my, 0.5f) : my;
  const float2 ef = f2((float)(((ix >> 23) & 0xff) - 127 + (hx ? 1 : 0)),
                       (float)(((iy >> 23) & 0xff) - 127 + (hy ? 1 : 0)));
  const float2 f = add2(f2(mx, my), f2b(-1.0f));
  const float2 s = mul2(f, own_rcpf2(add2(f2b(2.0f), f)));
  const float2 s2 = mul2(s, s);
  float2 p = f2b(1.0f / 11.0f);
  p = fma2(p, s2, f2b(1.0f / 9.0f));
  p = fma2(p, s2, f2b(1.0f / 7.0f));
  p = fma2(p, s2, f2b(1.0f / 5.0f));
  p = fma2(p, s2, f2b(1.0f / 3.0f));
  const float2 two_s = mul2(f2b(2.0f), s);
  const float2 lnm = fma2(mul2(two_s, s2), p, two_s);
  const float l2hi = 0.30102999566398120f;
  const float l2lo = (float)(0.30102999566398120 - (double)0.30102999566398120f);
  return fma2(ef, f2b(l2hi), fma2(ef, f2b(l2lo), mul2(lnm, f2b(0.43429448190325182f))));
}

// Dot2::add and Dot2::add_pair of N taps at once, in order: what does not depend
// on the sums first, then their chain, the errors, and the chain of those.  (One
// after another the ~12 dependent operations of a tap cost 90 cycles.)
template <int N>
__device__ __forceinline__ void dot2_taps(Dot2& acc, const float (&b)[N], const float (&x)[N]) {
  float p[N], t[N];
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = __fmul_rn(b[i], x[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) t[i] = __fadd_rn(i ? t[i - 1] : acc.s, p[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float a = i ? t[i - 1] : acc.s;
    const float q = __fmaf_rn(b[i], x[i], -p[i]);
    const float z = __fsub_rn(t[i], a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(t[i], z)), __fsub_rn(p[i], z));
    acc.c = __fadd_rn(acc.c, __fadd_rn(e, q));
  }
  acc.s = t[N - 1];
}
template <int N>
__device__ __forceinline__ void dot2_pairs(Dot2& acc, const float (&b)[N], const float (&x1)[N],
                                           const float (&x2)[N]) {
  float sg[N], p[N], t[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    sg[i] = __fadd_rn(x1[i], x2[i]);
    p[i] = __fmul_rn(b[i], sg[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) t[i] = __fadd_rn(i ? t[i - 1] : acc.s, p[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float zz = __fsub_rn(sg[i], x1[i]);
    const float ep = __fadd_rn(__fsub_rn(x1[i], __fsub_rn(sg[i], zz)), __fsub_rn(x2[i], zz));
    const float a = i ? t[i - 1] : acc.s;
    const float q = __fmaf_rn(b[i], sg[i], -p[i]);
    const float z = __fsub_rn(t[i], a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(t[i], z)), __fsub_rn(p[i], z));
    acc.c = __fadd_rn(acc.c, __fadd_rn(e, q));
    acc.c = __fmaf_rn(b[i], ep, acc.c);
  }
  acc.s = t[N - 1];
}

// The next N taps (tap pairs) of a point whose rows and taps lie one to a lane,
// from lane q on; N.
template <int N>
__device__ __forceinline__ int lane_taps(Dot2& acc, float b, float u, int q) {
  float gb[N], gu[N];
#pragma unroll
  for (int e = 0; e < N; ++e) {
    gb[e] = __shfl_sync(kFull, b, q + e);
    gu[e] = __shfl_sync(kFull, u, q + e);
  }
  dot2_taps(acc, gb, gu);
  return N;
}
// Dot2 of a point with all taps of a symmetric filter (fir_row_sym's order), by a
// warp: what is no chain by a lane per tap pair (rows and taps fetched at once, the
// pair's sum and product with their errors, later the error of its addition), and
// the chain of the rounded sums and then that of the errors by all lanes alike, from
// shared memory.  A pair costs 5 instructions and 12 cycles of a chain; all lanes
// doing all of it from shuffled values took 23 and 33.  The value of the point's own
// row in lane 0.
__device__ __forceinline__ float sym_point(Dot2& acc, const float* __restrict__ src,
                                           const float* TP, int n, PointScratch& W, int lane) {
  constexpr int kPer = kPairs / 32;
  const int half = n / 2;
  float p[kPer], q[kPer], own;
  {
    float x1[kPer], x2[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int k = lane + 32 * i;
      x1[i] = k < half ? __ldg(src - k * 256) : 0.0f;
      x2[i] = k < half ? __ldg(src - (n - 1 - k) * 256) : 0.0f;
    }
    own = x1[0];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int k = lane + 32 * i;
      const float b = k < half ? TP[k] : 0.0f;
      const float sg = __fadd_rn(x1[i], x2[i]);
      const float zz = __fsub_rn(sg, x1[i]);
      p[i] = __fmul_rn(b, sg);
      q[i] = __fmaf_rn(b, sg, -p[i]);
      W.p[k] = p[i];
      W.ep[k] = __fadd_rn(__fsub_rn(x1[i], __fsub_rn(sg, zz)), __fsub_rn(x2[i], zz));
    }
  }
  __syncwarp();
  float t = acc.s;
#pragma unroll 1
  for (int k = 0; k < half; k += 16) {
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = *reinterpret_cast<const float4*>(&W.p[k + 4 * j]);
    if (k + 16 <= half) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j].x = t = __fadd_rn(t, v[j].x);
        v[j].y = t = __fadd_rn(t, v[j].y);
        v[j].z = t = __fadd_rn(t, v[j].z);
        v[j].w = t = __fadd_rn(t, v[j].w);
      }
    } else {
      const int left = half - k;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j].x = t = 4 * j < left ? __fadd_rn(t, v[j].x) : t;
        v[j].y = t = 4 * j + 1 < left ? __fadd_rn(t, v[j].y) : t;
        v[j].z = t = 4 * j + 2 < left ? __fadd_rn(t, v[j].z) : t;
        v[j].w = t = 4 * j + 3 < left ? __fadd_rn(t, v[j].w) : t;
      }
    }
    __syncwarp();
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(&W.p[k + 4 * j]) = v[j];
    }
  }
  __syncwarp();
  float g[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int k = lane + 32 * i;
    const float to = W.p[k], a = k ? W.p[k - 1] : acc.s;
    const float z = __fsub_rn(to, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(to, z)), __fsub_rn(p[i], z));
    g[i] = __fadd_rn(e, q[i]);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kPer; ++i) W.p[lane + 32 * i] = g[i];
  __syncwarp();
  float c = acc.c;
  int k = 0;
#pragma unroll 1
  for (; k + 8 <= half; k += 8) {
    float b[8];
    float4 g4[2], e4[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      g4[j] = *reinterpret_cast<const float4*>(&W.p[k + 4 * j]);
      e4[j] = *reinterpret_cast<const float4*>(&W.ep[k + 4 * j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) b[j] = TP[k + j];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      c = __fmaf_rn(b[4 * j], e4[j].x, __fadd_rn(c, g4[j].x));
      c = __fmaf_rn(b[4 * j + 1], e4[j].y, __fadd_rn(c, g4[j].y));
      c = __fmaf_rn(b[4 * j + 2], e4[j].z, __fadd_rn(c, g4[j].z));
      c = __fmaf_rn(b[4 * j + 3], e4[j].w, __fadd_rn(c, g4[j].w));
    }
  }
  for (; k < half; ++k) c = __fmaf_rn(TP[k], W.ep[k], __fadd_rn(c, W.p[k]));
  __syncwarp();  // (the scratch is free)
  acc.s = t;
  acc.c = c;
  if (n & 1) acc.add(TP[half], __ldg(src - half * 256));
  return own;
}

// Dot2 of one output in the orders of ihc_lambda.cu (fir_row, fir_row_sym),
// rows of 256 sections in global memory; src points at the output's row.
__device__ __forceinline__ float dot2_row(const float* __restrict__ src,
                                          const float* __restrict__ taps_b, int taps, int n,
                                          bool sym) {
  constexpr int kBatch = 8;
  Dot2 acc;
  acc.init();
  if (sym && taps == n) {
    const float* far = src - (int64_t)(n - 1) * 256;
    const int half = n / 2, whole = half / kBatch * kBatch;
    for (int k0 = 0; k0 < whole; k0 += kBatch) {
      float b[kBatch], u[kBatch], w[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        u[i] = __ldg(src - (k0 + i) * 256);
        w[i] = __ldg(far + (k0 + i) * 256);
        b[i] = taps_b[k0 + i];
      }
      dot2_pairs(acc, b, u, w);
    }
    for (int k = whole; k < half; ++k)
      acc.add_pair(taps_b[k], __ldg(src - k * 256), __ldg(far + k * 256));
    if (n & 1) acc.add(taps_b[half], __ldg(src - half * 256));
  } else {
    const int whole = taps / kBatch * kBatch;
    for (int i0 = 0; i0 < whole; i0 += kBatch) {
      float b[kBatch], u[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        u[i] = __ldg(src - (i0 + i) * 256);
        b[i] = taps_b[i0 + i];
      }
      dot2_taps(acc, b, u);
    }
    for (int i = whole; i < taps; ++i) acc.add(taps_b[i], __ldg(src - i * 256));
  }
  return acc.result();
}

// Dot2 of eight rows with all n taps each, in the orders of dot2_row, a section to a
// lane; src points at the first row.  Rows r and r + 4 form pair r (fir_block8 and
// fir_block8_sym of ihc_lambda.cu); the rows of the next four taps are fetched while
// four are added, since they come from L2.  The rows read lie in [0, 7] and, of the
// older ones, not past the last tap's.
__device__ __forceinline__ void dot2_block8(const float* __restrict__ src, const float* TP, int n,
                                         bool sym, float (&out)[8]) {
  constexpr int kAhead = 4;
  Dot2x2 acc[4];
  float2 W[4];
  const float* older = src - 256;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    acc[j].init();
    W[j] = f2(__ldg(src + j * 256), __ldg(src + (j + 4) * 256));
  }
  auto shift = [&](float u) {
    const float last = W[3].x;
    W[3] = W[2];
    W[2] = W[1];
    W[1] = W[0];
    W[0] = f2(u, last);
  };
  if (sym) {
    const float* far = src - (n - 1) * 256;
    float2 V[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) V[j] = f2(__ldg(far + j * 256), __ldg(far + (j + 4) * 256));
    far += 8 * 256;
    const int half = n / 2;
    float u[kAhead], w[kAhead];
    auto fetch = [&](int k) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        u[i] = __ldg(older - (k + i) * 256);
        w[i] = __ldg(far + (k + i) * 256);
      }
    };
    auto step = [&](int k, float un, float wn) {
      const float2 bk = f2b(TP[k]);
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j].add_pair(bk, W[j], V[j]);
      shift(un);
      const float next = V[0].y;
      V[0] = V[1];
      V[1] = V[2];
      V[2] = V[3];
      V[3] = f2(next, wn);
    };
    // (the last fetch reaches rows -half - 4 and half + 12 - n)
    static_assert(kTensorMinTaps / 2 >= 5, "rows fetched ahead stay inside the window");
    fetch(0);
    int k = 0;
#pragma unroll 1
    for (; k + kAhead <= half; k += kAhead) {
      float un[kAhead], wn[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        un[i] = u[i];
        wn[i] = w[i];
      }
      fetch(k + kAhead);
#pragma unroll
      for (int i = 0; i < kAhead; ++i) step(k + i, un[i], wn[i]);
    }
#pragma unroll
    for (int i = 0; i < kAhead - 1; ++i)
      if (k + i < half) step(k + i, u[i], w[i]);
    if (n & 1) {
      const float2 bc = f2b(TP[half]);
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j].add(bc, W[j]);
    }
  } else {
    float u[kAhead];
    auto fetch = [&](int k) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i) u[i] = __ldg(older - min(k + i, n - 2) * 256);
    };
    fetch(0);
#pragma unroll 1
    for (int k = 0; k < n; k += kAhead) {
      float un[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) un[i] = u[i];
      fetch(k + kAhead);
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        if (k + i < n) {
          const float2 b = f2b(TP[k + i]);
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[j].add(b, W[j]);
        }
        shift(un[i]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 r = acc[j].result();
    out[j] = r.x;
    out[j + 4] = r.y;
  }
}

// Adds N values to s + c by TwoSum, in order: the chain of rounded sums first,
// then their errors, which do not depend on each other, then the chain of those.
template <int N>
__device__ __forceinline__ void two_sum_chain(float& s, float& c, const float (&x)[N]) {
  float t[N];
  t[0] = __fadd_rn(s, x[0]);
#pragma unroll
  for (int q = 1; q < N; ++q) t[q] = __fadd_rn(t[q - 1], x[q]);
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const float a = q ? t[q - 1] : s;
    const float z = __fsub_rn(t[q], a);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(a, __fsub_rn(t[q], z)), __fsub_rn(x[q], z)));
  }
  s = t[N - 1];
}

// Eight rows of a full window: row q adds x[2q] and x[2q + 1] to s + c, whose
// values after it are rs[q], rc[q].
__device__ __forceinline__ void two_sum_rows(float& s, float& c, const float (&x)[16],
                                             float (&rs)[8], float (&rc)[8]) {
  float t[16];
  t[0] = __fadd_rn(s, x[0]);
#pragma unroll
  for (int q = 1; q < 16; ++q) t[q] = __fadd_rn(t[q - 1], x[q]);
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const float a = q ? t[q - 1] : s;
    const float z = __fsub_rn(t[q], a);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(a, __fsub_rn(t[q], z)), __fsub_rn(x[q], z)));
    if (q & 1) {
      rs[q >> 1] = t[q];
      rc[q >> 1] = c;
    }
  }
  s = t[15];
}

// The DC window of `taps` rows that ends at ring row i, newest first, by TwoSum;
// the loads of sixteen rows ahead of their sums.  col: the section's column of
// the ring.
__device__ __forceinline__ void window_sum(const float* col, int i, int taps, int ring,
                                           float& ws, float& wc) {
  float s = 0.0f, c = 0.0f;
  while (taps > 0) {
    const int len = min(taps, i + 1);
    const float* p = col + i * kPitch;
    int j = 0;
    for (; j + 16 <= len; j += 16, p -= 16 * kPitch) {
      float u[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) u[q] = p[-q * kPitch];
      two_sum_chain(s, c, u);
    }
    for (; j < len; ++j, p -= kPitch) two_sum_add(s, c, *p);
    taps -= len;
    i = ring - 1;
  }
  ws = s;
  wc = c;
}

// Dot2 of a tile's rows (first frame row kb, before k_hi), a warp to eight rows and 32
// sections: of all, whose AC goes to ac[row][kPitch], or of those with a point in doubt and
// those that the products cannot give.  Eight rows with all taps together take 18k cycles
// of the FP32 pipe; a row for itself fetches its window from L2, which takes longer than
// its sums.  v: the frame's row 0 at the lane's section, col: that section's column.
// (Not inline: the loop over the tiles has no registers to spare.)
__device__ __noinline__ void ac_blocks(const TensorShared& S, const float* __restrict__ v,
                                       const cgb_ihc_frame& f, const float* TP, int n_ac,
                                       bool sym, int kb, int k_lo, int k_hi, bool all, int warp,
                                       float* ac, int col) {
  const int sg = warp & 1, gw = warp >> 1;
#pragma unroll 1
  for (int r0 = 8 * gw; r0 < tfir::kRows; r0 += 64) {
    const int k0 = kb + r0;
    uint32_t rows = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = r0 + i;
      if (k0 + i >= k_lo && k0 + i < k_hi &&
          (all || S.row[r] == kRowDot2 ||
           *reinterpret_cast<const uint32_t*>(&S.flag[r][4 * sg]) != 0))
        rows |= 1u << i;
    }
    const float* src = v + (int64_t)k0 * 256;
    const int sgm = k0 < f.frdp - 1 ? f.seg : f.total, lim = (k0 + 1) % sgm;
    const bool full = k0 + 8 <= k_hi && lim >= n_ac && lim + 7 < sgm &&
                      (k0 + 8 <= f.frdp - 1 || k0 >= f.frdp - 1);
    if (full && __popc(rows) >= 5) {
      float y[8];
      dot2_block8(src, TP, n_ac, sym, y);
#pragma unroll
      for (int i = 0; i < 8; ++i) ac[(r0 + i) * kPitch + col] = y[i];
    } else {
      for (; rows; rows &= rows - 1) {
        const int i = __ffs(rows) - 1;
        ac[(r0 + i) * kPitch + col] =
            dot2_row(src + i * 256, TP, taps_used(k0 + i, f, n_ac), n_ac, sym);
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads, 1)
    ihc_tensor_kernel(const IHCArgs A, const float* __restrict__ v,
                      const TensorTaps taps) {
  extern __shared__ __align__(128) unsigned char smem[];
  // layout: digits of x, two halves | band of the taps | dS, a ring of n_dc + 128
  // rows | AC [128] | taps with 128 zeros before and zeros up to 384 | TensorShared
  unsigned char* XD = smem;
  unsigned char* AD = XD + 2 * tfir::kHalfBytes;
  const int ring = A.n_dc + tfir::kRows;
  float* DS = reinterpret_cast<float*>(AD + tfir::kTapBytes);
  float* AC = DS + (size_t)ring * kPitch;
  float* TP = AC + (size_t)tfir::kRows * kPitch + tfir::kRows;  // zeros before and after
  TensorShared& S = *reinterpret_cast<TensorShared*>(
      (reinterpret_cast<uintptr_t>(TP + tfir::kDepth) + 15) & ~uintptr_t(15));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_ac = A.n_ac, n_dc = A.n_dc;

  // frame and run
  const int bx = blockIdx.x;
  int flo = 0, fhi = A.n_frames;
  while (fhi - flo > 1) {
    const int mid = (flo + fhi) >> 1;
    if (A.tile_prefix[mid] <= bx) flo = mid; else fhi = mid;
  }
  const cgb_ihc_frame f = A.frames[flo];
  const int tiles = (f.lam_rows + tfir::kRows - 1) / tfir::kRows;
  const int t0 = (bx - A.tile_prefix[flo]) * A.run;
  const int t1 = min(t0 + A.run, tiles);
  const int s0 = blockIdx.y * kCols;
  // the first output tile needs dS on the DC filter's look-back: whole tiles
  // before it, computed up to dS only
  const int back = min(t0, (n_dc - 1 + tfir::kRows - 1) / tfir::kRows);
  const int first = t0 - back;

  if (threadIdx.x == 0) {
    for (int h = 0; h < 2; ++h) {
      mbar_init(&S.mbar[h], 1);
      mbar_init(&S.ready[h], kIhcWarps);
    }
    mbar_init(&S.drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    S.abort = S.stop = 0;
    S.listed = S.late = 0;
    S.dot2_rows[0] = S.dot2_rows[1] = 0;
  }
  if (threadIdx.x < 2 * kCols) (&S.top[0][0])[threadIdx.x] = 0;
  if (threadIdx.x < kCols) S.partial[threadIdx.x] = 0;
  if (warp == kIhcWarps) tfir::tmem_alloc(&S.tmem);
  // taps, and the band of their digits (the digits of a tap pass through AC)
  uint16_t* td = reinterpret_cast<uint16_t*>(AC);
  for (int i = (int)threadIdx.x - tfir::kRows; i < tfir::kDepth; i += kThreads) {
    const float b = i >= 0 && i < n_ac ? A.taps[i] : 0.0f;
    TP[i] = b;
    if (i < 0 || i >= n_ac) continue;
    float r = b;
    float up = __int_as_float((127 + 8 - taps.exp_b) << 23);
    for (int j = 0; j < tfir::kDigits; ++j) {
      td[j * n_ac + i] = (uint16_t)(__float_as_uint(tfir::digit(r, up)) >> 16);
      up = 512.0f;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < tfir::kDigits * tfir::kCores * 64; e += kThreads) {
    const int j = e / (tfir::kCores * 64), q = e - j * (tfir::kCores * 64);
    const int i = 8 * (q >> 6) + ((q >> 3) & 7) + (q & 7) - (tfir::kRows - 1);
    reinterpret_cast<uint16_t*>(AD)[e] = i >= 0 && i < n_ac ? td[j * n_ac + i] : (uint16_t)0;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tfir::fence_before();
  __syncthreads();
  tfir::fence_after();
  const uint32_t tmem = __shfl_sync(kFull, S.tmem, 0);

  if (warp >= kIhcWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
  }
  if (warp == kIhcWarps) {
    // the issuing warp
    const uint32_t issue = tfir::elected();
    for (int n = 0;;) {  // digits so far
      for (int i = 0; i < tfir::kRowDigits; ++i, ++n) {
        for (int h = 0; h < 2; ++h) {
          if (!half_wait(S, h, n)) goto done;
          tfir::fence_after();
          // (test-only: the first half's products are left out, so that the
          // wait for them runs out)
          if (A.skip_first_copy && n == 0 && h == 0) continue;
          tfir::products(smem_u32(AD), smem_u32(XD) + h * tfir::kHalfBytes, tmem, i, h, issue);
          if (issue) tfir::commit(&S.mbar[h]);
          __syncwarp();
        }
      }
    }
  done:
    // The shared memory that the products read and the tensor memory that they write
    // are given up only after the last of them, also where nobody waited for it.
    if (issue) tfir::commit(&S.drained);
    const unsigned long long start = global_ns();
    while (!mbar_done(&S.drained, 0) && global_ns() - start < kWaitNs) {
    }
    __syncwarp();
  } else if (warp < kIhcWarps) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWorkerRegs));
    const int sg = warp & 1, gw = warp >> 1;  // section half; rows of x 24 gw .. of each half
    const int sec = 32 * sg + lane;           // this lane's section of the tile
    const float* vf = v + (int64_t)f.v_row0 * 256 + s0;

    // Rows of the tile whose sums the products can give: x is taken from row
    // kmin on (the first row of the segment, or of the first output's full
    // look-back), so a row qualifies if its own window starts there or has all
    // taps.  Others, in the tile where a segment ends, go to Dot2.  Called by
    // 128 threads and one (kmin).
    auto window_start = [&](int kb) {
      int k = kb;
      int tu = taps_used(k, f, n_ac);
      if (tu == 0) tu = taps_used(++k, f, n_ac);
      return k - tu + 1;
    };
    // (rows that the DC filter does not look back on count as rows without taps)
    const int needed = t0 * tfir::kRows - (n_dc - 1);
    auto classify = [&](int t, int r) {
      const int k = t * tfir::kRows + r;
      const int tu = k >= needed && k < f.lam_rows ? taps_used(k, f, n_ac) : 0;
      const int kmin = window_start(t * tfir::kRows);
      const bool fits = (tu == n_ac && k - n_ac + 1 >= kmin) || k - tu + 1 == kmin;
      S.row[r] = tu == 0 ? kRowZero : (fits ? kRowSum : kRowDot2);
      if (tu > 0 && !fits) S.dot2_rows[t & 1] = 1;
    };

    float x[2][3][8];  // the tile's rows: half, row group, row (from the newest)
    auto load_tile = [&](int t) {
      const int kb = t * tfir::kRows, kmin = S.kmin[t & 1],
                kmax = min(kb + tfir::kRows, f.lam_rows);
      // the newest row of the thread's first group, and the groups down from it
      const float* src = vf + (int64_t)(kb + tfir::kRows - 1 - 24 * gw) * 256 + sec;
      const bool whole = kmax == kb + tfir::kRows && kmin <= kb - 192;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          const int group = 24 * h + 3 * gw + g;
          const int top = kb + tfir::kRows - 1 - 8 * group;
          const float* row = src - (192 * h + 8 * g) * 256;
          if (whole && group < 40) {  // rows kb - 192 and up
#pragma unroll
            for (int c = 0; c < 8; ++c) x[h][g][c] = __ldg(row - c * 256);
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c)
              x[h][g][c] = top - c >= kmin && top - c < kmax ? __ldg(row - c * 256) : 0.0f;
          }
        }
    };
    // (its registers are free)
    auto clear_tile = [&]() {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 3; ++g)
#pragma unroll
          for (int c = 0; c < 8; ++c) x[h][g][c] = 0.0f;
    };
    // The sums of the tile's last and first row over this thread's two runs of
    // 24 rows, in tap order, with their largest partial sums.
    auto sample_runs = [&]() {
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          // the tap of the last row's first product; of the first row's, 127 less
          const int i0 = 192 * h + 24 * gw - (r ? tfir::kRows - 1 : 0);
          float sum = 0.0f, most = 0.0f;
#pragma unroll
          for (int q = 0; q < 24; ++q) {
            sum = __fmaf_rn(TP[i0 + q], x[h][q / 8][q % 8], sum);
            most = fmaxf(most, fabsf(sum));
          }
          S.sample[r][8 * h + gw][sec] = make_float2(sum, most);
        }
    };
    // The largest partial sum of a sampled row, from above: of the sums from
    // either end (a symmetric filter adds tap pairs from both).
    auto sampled_partial = [&](int r, int c) {
      float total = 0.0f, most = 0.0f, back = 0.0f;
#pragma unroll
      for (int i = 0; i < kRuns; ++i) total = __fadd_rn(total, S.sample[r][i][c].x);
      float at = 0.0f;
#pragma unroll
      for (int i = 0; i < kRuns; ++i) {
        const float2 q = S.sample[r][i][c];
        most = fmaxf(most, __fadd_rn(fabsf(at), q.y));
        back = fmaxf(back, __fadd_rn(fabsf(__fsub_rn(total, at)), q.y));
        at = __fadd_rn(at, q.x);
      }
      atomicMax(&S.partial[c], __float_as_uint(__fadd_rn(most, back)));
    };
    // one digit of one half: three 16-byte stores per thread
    auto put_digit = [&](int h, float up) {
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        float d[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) d[c] = tfir::digit(x[h][g][c], up);
        *reinterpret_cast<uint4*>(XD + h * tfir::kHalfBytes + (3 * gw + g) * tfir::kBlockBytes +
                                  sec * 16) =
            make_uint4(tfir::pack2(d[0], d[1]), tfir::pack2(d[2], d[3]), tfir::pack2(d[4], d[5]),
                       tfir::pack2(d[6], d[7]));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      half_ready(S, h, lane);
    };
    // Phase `n` of mbar[h].  Bounded; after a wait that ran out none waits, the
    // tile goes on with what is there and the run ends with it.
    auto wait_half = [&](int h, int n) {
      unsigned long long start = 0;
      while (!mbar_done(&S.mbar[h], n)) {
        if (*(volatile int*)&S.abort) break;
        if (start == 0) start = global_ns();
        if (global_ns() - start > kWaitNs) {
          *(volatile int*)&S.abort = 1;
          break;
        }
      }
    };
    auto next_digit = [&](int n) {
      wait_half(0, n);
      put_digit(0, 512.0f);
      wait_half(1, n);
      put_digit(1, 512.0f);
    };

    // AC and dS of row r and section c of the tile.  at: ring row of its first dS row.
    auto store_point = [&](int at, int r, int c, float ac, float own) {
      const float ms = __fmaf_rn(own, A.scale, -ac);
      int slot = at + r;
      slot -= slot >= ring ? ring : 0;
      AC[r * kPitch + c] = ac;
      DS[slot * kPitch + c] = __fmul_rn(ms, ms);
    };
    auto blocks = [&](int t, bool all, float* ac) {
      ac_blocks(S, vf + sec, f, TP, n_ac, A.ac_sym != 0, t * tfir::kRows, needed,
                min((t + 1) * tfir::kRows, f.lam_rows), all, warp, ac, sec);
    };
    // AC and dS of a tile from its AC.
    auto take_blocks = [&](int t, int at, const float* ac) {
      const int kb = t * tfir::kRows, rows = min(tfir::kRows, f.lam_rows - kb);
      for (int r = gw; r < rows; r += 8)
        store_point(at, r, sec, ac[r * kPitch + sec], __ldg(vf + (int64_t)(kb + r) * 256 + sec));
    };
    // The steps that finish a tile, each between two barriers of the workers.
    auto dot2_points = [&](int t, int at) {
      const int listed = S.listed, kb = t * tfir::kRows;
      if (listed <= kFewPoints) {
        // Few points: a warp to each, whose lanes fetch the point's rows and the
        // taps at once (one trip to L2 where a lane's own sequence of batches
        // takes sixteen).
        for (int p = warp; p < listed; p += kIhcWarps) {
          const int r = S.list[p] / kCols, c = S.list[p] % kCols;
          const float* src = vf + (int64_t)(kb + r) * 256 + c;
          const int taps = taps_used(kb + r, f, n_ac);
          Dot2 acc;
          acc.init();
          float own;  // lane 0: the point's own row
          if (A.ac_sym && taps == n_ac) {
            own = sym_point(acc, src, TP, n_ac, S.point[warp], lane);
          } else {
            // lane + 32 i: the row of that tap
            float u[9], b[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) {
              const int k = lane + 32 * i;
              u[i] = k < taps ? __ldg(src - k * 256) : 0.0f;
              b[i] = k < n_ac ? TP[k] : 0.0f;
            }
            own = u[0];
#pragma unroll
            for (int i = 0; i < 9; ++i)
#pragma unroll 1
              for (int q = 0; q < 32 && 32 * i + q < taps;) {
                const int left = taps - 32 * i - q;
                if (left >= 8)
                  q += lane_taps<8>(acc, b[i], u[i], q);
                else if (left >= 4)
                  q += lane_taps<4>(acc, b[i], u[i], q);
                else
                  q += lane_taps<1>(acc, b[i], u[i], q);
              }
          }
          const float ac = acc.result();
          if (lane == 0) store_point(at, r, c, ac, own);
        }
      }
      // first the rows that the products cannot give, and of more points than the
      // list holds the rows with any, a warp to 32 sections;
      // then single points, as few warps as hold them (what a warp's sequence
      // costs does not depend on its lanes), from the highest warp down
      const bool all = listed > kList;
      int row = all || S.dot2_rows[t & 1] ? gw : tfir::kRows;
      int p = (kIhcWarps - 1 - warp) * 32 + lane;
      while (true) {
        int r, c;
        if (row < tfir::kRows) {
          // of too many points for the list: the row's, as flagged
          uint32_t points = all ? *reinterpret_cast<const uint32_t*>(&S.flag[row][4 * sg]) : 0;
          if (S.row[row] == kRowDot2) points = ~0u;
          r = row;
          c = sec;
          row += 8;
          if (!(points >> lane & 1)) continue;
        } else {
          if (all || listed <= kFewPoints || p >= listed) break;
          r = S.list[p] / kCols;
          c = S.list[p] % kCols;
          p += kWorkers;
        }
        const float* src = vf + (int64_t)(kb + r) * 256 + c;
        store_point(at, r, c,
                    dot2_row(src, TP, taps_used(kb + r, f, n_ac), n_ac, A.ac_sym != 0),
                    __ldg(src));
      }
    };
    // DC sums of ihc_lambda.cu's kernel: a warp per 32 rows and section half
    auto dc_sums = [&](int t, int at) {
      if (warp >= 4 * kGroups) return;
      const float d = A.taps[n_ac];  // uniform DC taps
      const int row0 = t * tfir::kRows, k_hi = min(row0 + tfir::kRows, f.lam_rows);
      const int kb = row0 + gw * kDcAnchor, ke = min(kb + kDcAnchor, k_hi);
      const float* col = DS + sec;
      auto pre = [&](float ws, float wc, float ac) {
        const float p = __fmul_rn(d, ws);
        const float q = __fmaf_rn(d, ws, -p);
        const float dc = __fadd_rn(p, __fmaf_rn(d, wc, q));
        return __fmaf_rn(ac, A.eta_ac, __fmul_rn(dc, A.eta_dc));
      };
      if (kb >= ke) return;
      int now = at + (kb - row0);  // ring row of k
      now -= now >= ring ? ring : 0;
      int sgm = kb < f.frdp - 1 ? f.seg : f.total;
      int lim = (kb + 1) % sgm;
      float* slot = AC + (kb - row0) * kPitch + sec;
      float ws, wc;
      if (ke - kb == kDcAnchor && lim >= n_dc && lim + kDcAnchor - 1 < sgm &&
          (ke <= f.frdp - 1 || kb >= f.frdp - 1)) {
        // every row of the block has the full window
        window_sum(col, now, n_dc, ring, ws, wc);
        slot[0] = pre(ws, wc, slot[0]);
        int old = now >= n_dc ? now - n_dc : now - n_dc + ring;
        // eight rows at a time (the first of them done)
#pragma unroll 1
        for (int r0 = 0; r0 < kDcAnchor; r0 += 8) {
          float un[8], uo[8], ac[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            un[q] = col[now * kPitch];
            uo[q] = col[old * kPitch];
            ac[q] = slot[q * kPitch];
            now = now + 1 == ring ? 0 : now + 1;
            old = old + 1 == ring ? 0 : old + 1;
          }
          // the block's first row is done: adding and removing nothing keeps it
          if (r0 == 0) un[0] = uo[0] = 0.0f;
          float y[16], tw[8], tc[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            y[2 * q] = un[q];
            y[2 * q + 1] = -uo[q];
          }
          two_sum_rows(ws, wc, y, tw, tc);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (r0 + q > 0) slot[q * kPitch] = pre(tw[q], tc[q], ac[q]);
          slot += 8 * kPitch;
        }
        return;
      }
      ws = wc = 0.0f;
      int tu_prev = -1;
      for (int k = kb; k < ke; ++k) {
        const int tu = lim < n_dc ? lim : n_dc;
        if (k == kb || (tu != tu_prev && tu != tu_prev + 1)) {
          ws = wc = 0.0f;
          int i = now;
          for (int j = 0; j < tu; ++j) {
            two_sum_add(ws, wc, col[i * kPitch]);
            i = i == 0 ? ring - 1 : i - 1;
          }
        } else {
          two_sum_add(ws, wc, col[now * kPitch]);
          const int old = now >= tu ? now - tu : now - tu + ring;
          if (tu == tu_prev) two_sum_add(ws, wc, -col[old * kPitch]);
        }
        tu_prev = tu;
        if (k + 1 == f.frdp - 1) {
          sgm = f.total;
          lim = (k + 2) % sgm;
        } else if (++lim == sgm) {
          lim = 0;
        }
        *slot = pre(ws, wc, *slot);
        slot += kPitch;
        now = now + 1 == ring ? 0 : now + 1;
      }
    };
    // kEmitRows rows each from `from` on, `step` apart, before `to`
    auto emit = [&](int t, int from, int to, int step) {
      const int row0 = t * tfir::kRows, k_hi = min(row0 + to, f.lam_rows);
      const float dmg = __ldg(A.dmg + (size_t)f.ihc_profile * 256 + s0 + sec);
      const float a0 = __ldg(A.aihc + s0 + sec), a1 = __ldg(A.aihc + 256 + s0 + sec),
                  a2 = __ldg(A.aihc + 512 + s0 + sec);
      const bool sec0 = s0 + sec == 0;
      for (int kb = row0 + from; kb < k_hi; kb += step) {
        float lg[kEmitRows], l0[kEmitRows], l1[kEmitRows], l2[kEmitRows];
#pragma unroll
        for (int r = 0; r < kEmitRows; r += 2) {
          // (rows past the frame: what is there, not stored)
          const float* pre = AC + (kb + r - row0) * kPitch + sec;
          const float2 y = mul2(f2b(dmg), f2(pre[0], pre[kPitch]));
          const float2 g2 =
              own_log10f2(add2(f2(fmaxf(y.x, 0.0f), fmaxf(y.y, 0.0f)), f2b(1e-20f)));
          const float2 m0 = mul2(f2b(a0), g2), m1 = mul2(f2b(a1), g2), m2 = mul2(f2b(a2), g2);
          lg[r] = g2.x;
          lg[r + 1] = g2.y;
          l0[r] = sec0 ? A.spont0 : fminf(A.sat, fmaxf(m0.x, A.spont0));
          l1[r] = sec0 ? A.spont1 : fminf(A.sat, fmaxf(m1.x, A.spont1));
          l2[r] = sec0 ? A.spont2 : fminf(A.sat, fmaxf(m2.x, A.spont2));
          l0[r + 1] = sec0 ? A.spont0 : fminf(A.sat, fmaxf(m0.y, A.spont0));
          l1[r + 1] = sec0 ? A.spont1 : fminf(A.sat, fmaxf(m1.y, A.spont1));
          l2[r + 1] = sec0 ? A.spont2 : fminf(A.sat, fmaxf(m2.y, A.spont2));
        }
        const int64_t at = (f.lam_row0 + kb) * 256 + s0 + sec;
        const int64_t plane = A.lam_plane_rows * 256;
        float* out = A.lam + at;
#pragma unroll
        for (int r = 0; r < kEmitRows; ++r) {
          if (kb + r < k_hi) {
            out[r * 256] = l0[r];
            out[plane + r * 256] = l1[r];
            out[2 * plane + r * 256] = l2[r];
            if (A.ihc) A.ihc[at + r * 256] = lg[r];
            if (A.lam_host) {
              A.lam_host[at + r * 256] = l0[r];
              A.lam_host[plane + at + r * 256] = l1[r];
              A.lam_host[2 * plane + at + r * 256] = l2[r];
            }
          }
        }
      }
    };

    if (threadIdx.x == 0) S.kmin[first & 1] = window_start(first * tfir::kRows);
    sync_workers();
    load_tile(first);
    int n = 0;       // completed phases of each half's barrier
    int at = 0;      // ring row of the tile's first dS row
    int at_prev = 0; // and of the tile before
    bool pending = false;  // the tile before is to be finished
    // A tile with more points in doubt than the list holds, also among its last rows (at
    // the start of a segment only the first rows have them) is finished before the next
    // is begun; after two the next tiles take Dot2 for all points: three, then more each
    // time.
    auto crowded = [&]() { return S.listed > kList && S.late > kLate; };
    bool before = false;  // the last tile with products was such a one
    int direct = 0, next_direct = 0;
    for (int t = first;; ++t) {
      if (direct > 0 || t == t1 || (pending && crowded())) {
        clear_tile();
        if (pending) {
          if (S.listed > kList) {
            blocks(t - 1, false, AC);
            sync_workers();
            take_blocks(t - 1, at_prev, AC);
          } else {
            dot2_points(t - 1, at_prev);
          }
          sync_workers();
        }
        // A tile without products: the FP32 pipe is busy with its sums while half of the
        // warps first finish the tile before, 32 rows each.
        const bool own = direct > 0 && t < t1;
        float* const all = reinterpret_cast<float*>(XD);
        static_assert(tfir::kRows * kPitch * 4 <= 2 * tfir::kHalfBytes, "AC in the digits' place");
        if (pending && t > t0) {
          dc_sums(t - 1, at_prev);
          if (!own) sync_workers();
          if (!own || warp < 4 * kGroups)
            emit(t - 1, own ? kDcAnchor * gw : kEmitRows * gw,
                 own ? kDcAnchor * (gw + 1) : tfir::kRows, own ? kEmitRows : 8 * kEmitRows);
        }
        if (own) blocks(t, true, all);
        if (threadIdx.x == 0) {
          S.listed = S.late = 0;
          S.dot2_rows[t & 1] = S.dot2_rows[(t + 1) & 1] = 0;
          S.kmin[(t + 1) & 1] = window_start((t + 1) * tfir::kRows);
        }
        if (t == t1) break;
        if (own) {
          if (warp < kGroups && gw == 0) S.top[(t + 1) & 1][sec] = 0;
          sync_workers();
          take_blocks(t, at, all);
          if (--direct == 0 && t + 1 < t1) load_tile(t + 1);
          sync_workers();
          pending = true;
          at_prev = at;
          at += tfir::kRows;
          at -= at >= ring ? ring : 0;
          continue;
        }
        pending = false;
        load_tile(t);
        sync_workers();
      }
      const int kb = t * tfir::kRows, k_hi = min(kb + tfir::kRows, f.lam_rows);
      // scales: the exponent of the section's largest |x| (a NaN is not seen
      // here: it makes every sum of its section a NaN, which Dot2 then replaces)
      uint32_t* top = S.top[t & 1];
      {
        float m = 0.0f;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int c = 0; c < 8; ++c) m = fmaxf(m, fabsf(x[h][g][c]));
        atomicMax(&top[sec], __float_as_uint(m));
      }
      sample_runs();
      sync_workers();
      const uint32_t m = top[sec];
      const int e = (int)(m >> 23) - 126;  // 2^(e-1) <= largest |x| < 2^e
      // magnitudes whose digits and result are far from the ends of the FP32
      // range; an infinity has e = 129
      const bool usable = e >= -80 && e <= 100;
      if (warp < kGroups && gw == 0) {
        S.scale[sec] =
            make_float2(m == 0 ? 0.0f : (usable ? taps.floor : __int_as_float(0x7f800000)),
                        usable ? __int_as_float((127 + e + taps.exp_b - 16) << 23) : 1.0f);
        S.top[(t + 1) & 1][sec] = 0;
      }
      const float up = usable ? __int_as_float((127 + 8 - e) << 23) : 0.0f;
      if (!usable) clear_tile();  // (0 times an infinity is no digit)
      put_digit(0, up);
      put_digit(1, up);
      if (warp >= 8 && warp < 12) sampled_partial((warp >> 1) & 1, 32 * (warp & 1) + lane);
      sync_workers();
      // the tile before, between the digits of this one
      const bool prev_out = pending && t > t0;
      if (pending) dot2_points(t - 1, at_prev);
      next_digit(n);
      sync_workers();
      if (threadIdx.x == 0) {
        S.listed = S.late = 0;
        S.dot2_rows[(t + 1) & 1] = 0;
        S.kmin[(t + 1) & 1] = window_start((t + 1) * tfir::kRows);
      }
      if (prev_out) dc_sums(t - 1, at_prev);
      if (warp >= 12) classify(t, (int)threadIdx.x - 384);
      next_digit(n + 1);
      sync_workers();
      // slack of the rounding test (head of the file)
      if (warp < kGroups && gw == 0) {
        S.scale[sec].x += __fdiv_rn(__uint_as_float(S.partial[sec]) * 0x1.4p-43f, S.scale[sec].y);
        S.partial[sec] = 0;
      }
      if (prev_out) emit(t - 1, gw * kEmitRows, tfir::kRows / 2, 8 * kEmitRows);
      next_digit(n + 2);
      if (prev_out)
        emit(t - 1, tfir::kRows / 2 + gw * kEmitRows, tfir::kRows, 8 * kEmitRows);
      next_digit(n + 3);
      // the row's velocity, for dS
      const int row = (warp & 3) * 32 + lane, cols = (warp >> 2) * 16;
      float4 own[4];
      {
        const float4* src =
            reinterpret_cast<const float4*>(vf + (int64_t)(kb + row) * 256 + cols);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          own[i] = kb + row < k_hi ? __ldg(src + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
      next_digit(n + 4);
      wait_half(0, n + 5);
      wait_half(1, n + 5);
      sync_workers();
      tfir::fence_after();

      // Epilogue: lane = row, sixteen sections per thread.  The digits' sum as
      // an unevaluated FP32 pair h + c, rounded once.
      {
        const int kind = S.row[row];
        int slot = at + row;
        slot -= slot >= ring ? ring : 0;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const int c0 = cols + part * 8;
          const uint32_t from = tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0;
          float G[tfir::kSums][8];
#pragma unroll
          for (int i = 0; i < tfir::kSums; ++i) tfir::tmem_load8(from + kCols * i, G[i]);
          tfir::tmem_wait_loads();
          uint32_t bad = 0;
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            const float2 q = f2b(1.0f / 512.0f);
            float2 g[tfir::kSums];
#pragma unroll
            for (int i = 0; i < tfir::kSums; ++i) g[i] = f2(G[i][c], G[i][c + 1]);
            float2 e2, e1, e0;
            const float2 g3 = fma2(fma2(g[5], q, g[4]), q, g[3]);
            const float2 h2 = two_sum2(g[2], mul2(g3, q), e2);
            const float2 h1 = two_sum2(g[1], mul2(h2, q), e1);
            const float2 h0 = two_sum2(g[0], mul2(h1, q), e0);
            const float2 lo = fma2(fma2(e2, q, e1), q, e0);
            const float2 res = add2(h0, lo);
            const float2 rest = sub2(lo, sub2(res, h0));
            const float4 sc = *reinterpret_cast<const float4*>(&S.scale[c0 + c]);
            const float2 slack = f2(sc.x, sc.z);
            float2 ac = mul2(res, f2(sc.y, sc.w));
            const float2 up = add2(res, add2(rest, slack)), down = add2(res, sub2(rest, slack));
            const float least = 1e-30f;  // (far from where the unit's product would round)
            if (!(up.x == res.x && down.x == res.x && (sc.x == 0.0f || fabsf(ac.x) > least)) ||
                fmaxf(fmaxf(fabsf(g[2].x), fabsf(g[3].x)), fabsf(g[4].x)) >= taps.limit)
              bad |= 1u << c;
            if (!(up.y == res.y && down.y == res.y && (sc.z == 0.0f || fabsf(ac.y) > least)) ||
                fmaxf(fmaxf(fabsf(g[2].y), fabsf(g[3].y)), fabsf(g[4].y)) >= taps.limit)
              bad |= 2u << c;
            if (kind == kRowZero) ac = f2b(0.0f);
            const float4 o = own[2 * part + c / 4];
            const float2 ms = fma2(c & 2 ? f2(o.z, o.w) : f2(o.x, o.y), f2b(A.scale), neg2(ac));
            const float2 ds = mul2(ms, ms);
            AC[row * kPitch + c0 + c] = ac.x;
            AC[row * kPitch + c0 + c + 1] = ac.y;
            DS[slot * kPitch + c0 + c] = ds.x;
            DS[slot * kPitch + c0 + c + 1] = ds.y;
          }
          if (kind != kRowSum) bad = 0;
          S.flag[row][c0 >> 3] = (unsigned char)bad;
          if (bad) {
            int p = atomicAdd(&S.listed, __popc(bad));
            if ((warp & 3) == 3) atomicAdd(&S.late, __popc(bad));
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (bad >> c & 1) {
                if (p < kList) S.list[p] = (uint16_t)(row * kCols + c0 + c);
                ++p;
              }
          }
        }
      }
      if (t + 1 < t1) load_tile(t + 1);
      tfir::fence_before();
      sync_workers();
      at_prev = at;
      at += tfir::kRows;
      at -= at >= ring ? ring : 0;
      if (*(volatile int*)&S.abort) {
        if (threadIdx.x == 0) atomicOr(A.status, 1);
        break;
      }
      pending = true;
      n += tfir::kRowDigits;
      const bool now = crowded();
      next_direct = now && before ? min(2 * next_direct + 3, kDirectTiles) : 0;
      direct = next_direct;
      before = now;
    }
    if (threadIdx.x == 0) *(volatile int*)&S.stop = 1;
  }
  __syncthreads();
  if (warp == kIhcWarps) tfir::tmem_free(tmem);
}

size_t tensor_smem(int n_dc) {
  return 2 * (size_t)tfir::kHalfBytes + tfir::kTapBytes +
         ((size_t)n_dc + 2 * tfir::kRows) * kPitch * 4 + (size_t)(tfir::kRows + tfir::kDepth) * 4 + 16 +
         sizeof(TensorShared);
}

}  // namespace

bool ihc_tensor_fits(int n_ac, int n_dc) {
  return n_ac >= kTensorMinTaps && n_ac <= tfir::kMaxTaps &&
         tensor_smem(n_dc) <= 227 * 1024;
}

bool ihc_tensor_taps(const float* taps, int n_ac, float scale, TensorTaps* out) {
  float top = 0.0f;
  for (int i = 0; i < n_ac; ++i) {
    const float b = taps[i] * scale;
    if (!std::isfinite(b)) return false;
    top = std::fmax(top, std::fabs(b));
  }
  if (!(top > 0.0f)) return false;
  std::frexp(top, &out->exp_b);
  if (out->exp_b < -16 || out->exp_b > 16) return false;
  // the digits as the kernel forms them (exactly), their sums and what they leave; in
  // units of 2^exp_b
  double S[tfir::kDigits] = {}, sum = 0.0, left = 0.0;
  for (int i = 0; i < n_ac; ++i) {
    double y = std::ldexp((double)(taps[i] * scale), 8 - out->exp_b);
    sum += std::fabs(y) / 256;
    for (int j = 0; j < tfir::kDigits; ++j) {
      const double d = std::nearbyint(y);
      S[j] += std::fabs(d);
      y = (y - d) * 512;
    }
    left += std::ldexp(std::fabs(y), -8 - 9 * tfir::kDigits);
  }
  // M_m of tensor_fir.cuh: digit i of x is at most 256
  double M[tfir::kSums];
  for (int m = 0; m < tfir::kSums; ++m) {
    M[m] = 0.0;
    for (int j = 0; j < tfir::kDigits && j <= m; ++j) M[m] += 256 * S[j];
  }
  const double exact = 0x1p24;
  const double most = std::fmax(M[2], std::fmax(M[3], M[4]));
  // (with random digits the accumulators have a standard deviation of 2^19.5)
  if (M[1] >= exact || most > 2 * exact - 0x1p22) return false;
  // What an accumulator of partial sums up to M may lose: at most 17 addends in each of
  // 18 steps of a digit pair, each cut to a multiple of 2^q.
  auto lost = [&](int pairs, double m) {
    const int q = m < exact ? 0 : (int)std::floor(std::log2(m / exact)) + 1;
    return 17.0 * 18.0 * pairs * (std::ldexp(1.0, q) - 1.0);
  };
  out->limit = most < exact ? std::numeric_limits<float>::infinity()
                            : (float)(2 * exact - most - lost(5, most));
  out->floor = (float)(1.01 * (std::ldexp(sum, 16 - 54) + std::ldexp(left, 16) +
                               std::ldexp(256 * (S[1] + S[2] + S[3] + S[4]), -54) +
                               std::ldexp(lost(5, M[5]), -45) +
                               0x1p-28));  // (and the rounding of g3 in the epilogue)
  return true;
}

int ihc_tensor_launch(const IHCArgs& A, const float* d_v, int n_runs, const TensorTaps& taps,
                      cudaStream_t st) {
  const size_t smem = tensor_smem(A.n_dc);
  CGB_TRY_CUDA(cudaFuncSetAttribute(ihc_tensor_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "cudaFuncSetAttribute(ihc tensor smem)");
  ihc_tensor_kernel<<<dim3((unsigned)n_runs, 256 / kCols), kThreads, smem, st>>>(A, d_v, taps);
  CGB_TRY_CUDA(cudaGetLastError(), "ihc_tensor_kernel launch");
  note_launch();
  return CGB_OK;
}

}  // namespace cgb
