// IHC + lambda with the AC filter on the tensor cores: the same stage as
// ihc_lambda.cu's kernel, bit for bit, for filters of up to 257 taps.
//
// What bounded the stage: 127 tap pairs of compensated FP32 arithmetic per
// point, ~2,170 lane operations (43 ms of the FP32 pipe on 2.9 million rows).
// Here the filter is a product of digit matrices (tensor_fir.cuh) that is exact
// to about 2^-41 of the scales, 17.6k cycles of the tensor pipe for a tile of
// 128 rows x 64 sections; 15 exact integers per point leave TMEM as five sums.
//
// The same bits as the compensated FIR (Dot2).  Both are the sum rounded once,
// up to errors far below an ulp: Dot2's stay under 2^-37.9 of (largest |x| of
// the window x largest |b|) over 2.8 million points of solved velocity (tones of
// 20-100 dB, noise of 0-40 dB), the digits' about 2^-41.  So the two can only
// differ where the exact sum lies that close to a rounding boundary.  The
// epilogue rounds sum +- slack; where that makes a difference (1-2% of the points
// of noisy signals, next to none of others), and in rows whose look-back is
// shorter than the tile's, the point is evaluated by Dot2 itself.
//
// One CTA: 64 sections x a run of tiles of one frame.  Sixteen warps hold the
// tile's 384 rows of velocity in registers (48 values a thread) and write one
// digit after another into two shared-memory halves; a seventeenth issues the
// products as soon as a half is there.  The first digit's products take a third
// of the tile's time, which the DC sums, IHC and lambda of the tile before pass
// under.
//
// Measured (GB300), against the FP32 pipe: JND sweep (2.9 million rows) 53.7 ->
// 25.9 ms, 176,000 rows in 33 intervals 4.46 -> 2.05 ms, one signal of 5,330 rows
// 0.80 -> 0.38 ms.

#include <cuda_runtime.h>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "ihc_common.cuh"
#include "ihc_tensor.h"
#include "tensor_fir.cuh"

namespace cgb {
namespace {

constexpr int kWorkers = kIhcWarps * 32;   // threads that do everything but issue
constexpr int kThreads = kWorkers + 128;   // the issuing warp's group of four
constexpr int kBarrier = kWorkers + 32;
// registers a thread: 96 at launch (640 threads), then 112 for the workers and
// 32 for the issuing warp's group, together the same
constexpr int kWorkerRegs = 112, kIssueRegs = 32;
static_assert(kWorkers * kWorkerRegs + 128 * kIssueRegs <= kThreads * 96, "register split");
constexpr int kCols = tfir::kCols;
constexpr int kPitch = kCols + 1;          // a row of dS / AC: lanes along rows too
constexpr int kGroups = kCols / 32;        // section halves

struct TensorShared {
  uint64_t mbar[2];          // products of half h are done
  uint32_t tmem;
  int abort;
  int listed;                // points for Dot2
  int listed_pad;
  uint32_t top[2][kCols];    // largest |x| bits of the tile, by tile parity
  float slack[kCols];        // in units of the accumulators; +inf: no usable scale
  float unit[kCols];         // 2^(e+eb-16)
};

__device__ __forceinline__ void sync_workers() {
  asm volatile("bar.sync 3, %0;" ::"n"(kWorkers) : "memory");
}
__device__ __forceinline__ void half_ready(int h) {  // workers
  asm volatile("bar.arrive %0, %1;" ::"r"(1 + h), "n"(kBarrier) : "memory");
}
__device__ __forceinline__ void half_wait(int h) {  // the issuing warp
  asm volatile("bar.sync %0, %1;" ::"r"(1 + h), "n"(kBarrier) : "memory");
}

// TwoSum
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float t = __fadd_rn(a, b);
  const float z = __fsub_rn(t, a);
  err = __fadd_rn(__fsub_rn(a, __fsub_rn(t, z)), __fsub_rn(b, z));
  return t;
}

// Dot2 of one output in the orders of ihc_lambda.cu (fir_row, fir_row_sym),
// rows of 256 sections in global memory; src points at the output's row.
__device__ float dot2_row(const float* __restrict__ src, const float* __restrict__ b, int taps,
                          int n, bool sym) {
  Dot2 acc;
  acc.init();
  if (sym && taps == n) {
#pragma unroll 4
    for (int k = 0; k < n / 2; ++k)
      acc.add_pair(b[k], src[-(int64_t)k * 256], src[-(int64_t)(n - 1 - k) * 256]);
    if (n & 1) acc.add(b[n / 2], src[-(int64_t)(n / 2) * 256]);
  } else {
#pragma unroll 4
    for (int i = 0; i < taps; ++i) acc.add(b[i], src[-(int64_t)i * 256]);
  }
  return acc.result();
}

__global__ void __launch_bounds__(kThreads, 1)
    ihc_tensor_kernel(const IHCArgs A, const float* __restrict__ v, int exp_b, float slack) {
  extern __shared__ __align__(128) unsigned char smem[];
  // layout: digits of x, two halves | band of the taps | dS [n_dc + 128] | AC
  // [128] | taps | TensorShared
  unsigned char* XD = smem;
  unsigned char* AD = XD + 2 * tfir::kHalfBytes;
  float* DS = reinterpret_cast<float*>(AD + tfir::kTapBytes);
  float* AC = DS + (size_t)(A.n_dc + tfir::kRows) * kPitch;
  float* TP = AC + (size_t)tfir::kRows * kPitch;
  TensorShared& S = *reinterpret_cast<TensorShared*>(
      (reinterpret_cast<uintptr_t>(TP + A.n_ac) + 15) & ~uintptr_t(15));
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
    for (int h = 0; h < 2; ++h)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.mbar[h])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    S.abort = 0;
    S.listed = 0;
  }
  if (threadIdx.x < 2 * kCols) (&S.top[0][0])[threadIdx.x] = 0;
  if (warp == kIhcWarps) tfir::tmem_alloc(&S.tmem);
  // taps, and the band of their digits (the digits of a tap pass through AC)
  uint16_t* td = reinterpret_cast<uint16_t*>(AC);
  for (int i = threadIdx.x; i < n_ac; i += kThreads) {
    const float b = A.taps[i];
    TP[i] = b;
    float r = b;
    float up = __int_as_float((127 + 8 - exp_b) << 23);
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
    bool run = true;
    for (int t = first; t < t1 && run; ++t) {
      for (int i = 0; i < tfir::kDigits && run; ++i) {
        for (int h = 0; h < 2; ++h) {
          half_wait(h);
          if (*(volatile int*)&S.abort) {
            run = false;
            break;
          }
          tfir::fence_after();
          // (test-only: the first half's products are left out, so that the
          // wait for them runs out)
          if (A.skip_first_copy && t == first && i == 0 && h == 0) continue;
          tfir::products(smem_u32(AD), smem_u32(XD) + h * tfir::kHalfBytes, tmem, i, h, issue);
          if (issue) tfir::commit(&S.mbar[h]);
          __syncwarp();
        }
      }
    }
  } else if (warp < kIhcWarps) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWorkerRegs));
    const int sg = warp & 1, gw = warp >> 1;  // section half; row groups gw, gw + 8, ...
    const int sec = 32 * sg + lane;           // this lane's section of the tile
    const float dmg = A.dmg[(size_t)f.ihc_profile * 256 + s0 + sec];
    const float a0 = A.aihc[0 * 256 + s0 + sec], a1 = A.aihc[1 * 256 + s0 + sec],
                a2 = A.aihc[2 * 256 + s0 + sec];
    const bool sec0 = s0 + sec == 0;
    const float* vf = v + (int64_t)f.v_row0 * 256 + s0;

    // Rows of the tile at kb whose sums the products can give: x is taken from
    // row kmin on (the first row of the segment, or of the first output's full
    // look-back), so a row qualifies if its own window starts there or has all
    // taps.  Others, in the tile where a segment ends, go to Dot2.
    auto window_start = [&](int kb) {
      int k = kb;
      int tu = taps_used(k, f, n_ac);
      if (tu == 0) tu = taps_used(++k, f, n_ac);
      return k - tu + 1;
    };

    float x[2][3][8];  // the tile's rows: half, row group, row (from the newest)
    auto load_tile = [&](int t) {
      const int kb = t * tfir::kRows, kmin = window_start(kb),
                kmax = min(kb + tfir::kRows, f.lam_rows);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          const int top = kb + tfir::kRows - 1 - 8 * (24 * h + gw + 8 * g);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int k = top - c;
            x[h][g][c] = k >= kmin && k < kmax ? __ldg(vf + (int64_t)k * 256 + sec) : 0.0f;
          }
        }
    };
    // one digit of one half: three 16-byte stores per thread
    auto put_digit = [&](int h, float up) {
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        float d[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) d[c] = tfir::digit(x[h][g][c], up);
        *reinterpret_cast<uint4*>(XD + h * tfir::kHalfBytes + (gw + 8 * g) * tfir::kBlockBytes +
                                  sec * 16) =
            make_uint4(tfir::pack2(d[0], d[1]), tfir::pack2(d[2], d[3]), tfir::pack2(d[4], d[5]),
                       tfir::pack2(d[6], d[7]));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      half_ready(h);
    };
    // phase `n` of mbar[h], bounded; false: every worker gives up
    auto wait_half = [&](int h, int n) {
      uint32_t done = 0;
      const unsigned long long start = global_ns();
      while (!done) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_u32(&S.mbar[h])), "r"((uint32_t)(n & 1))
            : "memory");
        if (!done && global_ns() - start > kWaitNs) break;
      }
      if (!done) *(volatile int*)&S.abort = 1;
      sync_workers();
      return *(volatile int*)&S.abort == 0;
    };

    // DC sums, IHC and lambda of tile t (dS and AC in shared memory): phase 2
    // of ihc_lambda.cu's kernel.
    auto finish_tile = [&](int t) {
      const int row0 = t * tfir::kRows, k_hi = min(row0 + tfir::kRows, f.lam_rows);
      const int dsbase = row0 - n_dc;
      const float d = A.taps[n_ac];  // uniform DC taps
      if (warp < 4 * kGroups) {
        const int kb = row0 + (warp >> 1) * kDcAnchor;
        const int ke = min(kb + kDcAnchor, k_hi);
        const float* col = DS + sec;
        float ws = 0.0f, wc = 0.0f;
        int tu_prev = -1;
        int sgm = kb < f.frdp - 1 ? f.seg : f.total;
        int lim = (kb + 1) % sgm;
#pragma unroll 4
        for (int k = kb; k < ke; ++k) {
          const int tu = lim < n_dc ? lim : n_dc;
          const float x_new = col[(k - dsbase) * kPitch];
          const float x_old = col[(k - tu - dsbase) * kPitch];
          if (k == kb || (tu != tu_prev && tu != tu_prev + 1)) {
            ws = wc = 0.0f;
            for (int j = 0; j < tu; ++j) two_sum_add(ws, wc, col[(k - j - dsbase) * kPitch]);
          } else {
            two_sum_add(ws, wc, x_new);
            if (tu == tu_prev) two_sum_add(ws, wc, -x_old);
          }
          tu_prev = tu;
          if (k + 1 == f.frdp - 1) {
            sgm = f.total;
            lim = (k + 2) % sgm;
          } else if (++lim == sgm) {
            lim = 0;
          }
          const float p = __fmul_rn(d, ws);
          const float q = __fmaf_rn(d, ws, -p);
          const float dc = __fadd_rn(p, __fmaf_rn(d, wc, q));
          float& slot = AC[(k - row0) * kPitch + sec];
          slot = __fmaf_rn(slot, A.eta_ac, __fmul_rn(dc, A.eta_dc));
        }
      }
      sync_workers();
      for (int kb = row0 + gw * kEmitRows; kb < k_hi; kb += 8 * kEmitRows) {
        float lg[kEmitRows], l0[kEmitRows], l1[kEmitRows], l2[kEmitRows];
#pragma unroll
        for (int r = 0; r < kEmitRows; ++r) {
          const int k = min(kb + r, k_hi - 1);
          const float y = __fmul_rn(dmg, AC[(k - row0) * kPitch + sec]);
          lg[r] = own_log10f(__fadd_rn(fmaxf(y, 0.0f), 1e-20f));
          l0[r] = sec0 ? A.spont0 : fminf(A.sat, fmaxf(__fmul_rn(a0, lg[r]), A.spont0));
          l1[r] = sec0 ? A.spont1 : fminf(A.sat, fmaxf(__fmul_rn(a1, lg[r]), A.spont1));
          l2[r] = sec0 ? A.spont2 : fminf(A.sat, fmaxf(__fmul_rn(a2, lg[r]), A.spont2));
        }
#pragma unroll
        for (int r = 0; r < kEmitRows; ++r) {
          if (kb + r < k_hi) {
            const int64_t at = (f.lam_row0 + kb + r) * 256 + s0 + sec;
            const int64_t plane = A.lam_plane_rows * 256;
            A.lam[at] = l0[r];
            A.lam[plane + at] = l1[r];
            A.lam[2 * plane + at] = l2[r];
            if (A.ihc) A.ihc[at] = lg[r];
            if (A.lam_host) {
              A.lam_host[at] = l0[r];
              A.lam_host[plane + at] = l1[r];
              A.lam_host[2 * plane + at] = l2[r];
            }
          }
        }
      }
      sync_workers();
    };
    // dS of the next tile's look-back: n_dc rows down by a tile, in steps that
    // do not overlap
    auto shift_ds = [&]() {
      for (int i0 = 0; i0 < n_dc; i0 += tfir::kRows) {
        const int i1 = min(i0 + tfir::kRows, n_dc);
        for (int i = i0 + gw; i < i1; i += 8)
          DS[i * kPitch + sec] = DS[(i + tfir::kRows) * kPitch + sec];
        sync_workers();
      }
    };

    load_tile(first);
    bool ok = true;
    int n = 0;  // completed phases of each half's barrier
    for (int t = first; t < t1; ++t, n += tfir::kDigits) {
      const int kb = t * tfir::kRows, k_hi = min(kb + tfir::kRows, f.lam_rows);
      // scales: the exponent of the section's largest |x|
      uint32_t* top = S.top[t & 1];
      {
        uint32_t m = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int c = 0; c < 8; ++c)
              m = max(m, __float_as_uint(x[h][g][c]) & 0x7fffffffu);
        atomicMax(&top[sec], m);
      }
      sync_workers();
      const uint32_t m = top[sec];
      const int e = (int)(m >> 23) - 126;  // 2^(e-1) <= largest |x| < 2^e
      // magnitudes whose digits and result are far from the ends of the FP32
      // range; infinities and NaN have e = 129
      const bool usable = e >= -80 && e <= 100;
      if (threadIdx.x < kCols) {
        const uint32_t mm = top[threadIdx.x];
        const int ee = (int)(mm >> 23) - 126;
        const bool uu = ee >= -80 && ee <= 100;
        S.slack[threadIdx.x] = mm == 0 ? 0.0f : (uu ? slack : __int_as_float(0x7f800000));
        S.unit[threadIdx.x] = uu ? __int_as_float((127 + ee + exp_b - 16) << 23) : 1.0f;
        S.top[(t + 1) & 1][threadIdx.x] = 0;
      }
      const float up = usable ? __int_as_float((127 + 8 - e) << 23) : 0.0f;
      if (!usable) {  // (0 times an infinity is no digit)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int c = 0; c < 8; ++c) x[h][g][c] = 0.0f;
      }
      put_digit(0, up);
      put_digit(1, up);
      if (t > first) {
        if (t > t0) finish_tile(t - 1);
        shift_ds();
      }
      for (int i = 1; i < tfir::kDigits && ok; ++i) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (ok && !(ok = wait_half(h, n + i - 1))) half_ready(h);  // wakes the issuing warp
          if (ok) put_digit(h, 512.0f);
        }
      }
      if (!ok) break;
      if (t + 1 < t1) load_tile(t + 1);
      ok = wait_half(0, n + tfir::kDigits - 1);
      if (ok) ok = wait_half(1, n + tfir::kDigits - 1);
      if (!ok) {
        if (t + 1 < t1) half_ready(0);
        break;
      }
      tfir::fence_after();

      // Epilogue: lane = row, sixteen sections per thread.  The digits' sum as
      // an unevaluated FP32 pair h + c, rounded once.
      uint16_t* list = reinterpret_cast<uint16_t*>(XD);  // free until the next digit
      {
        const int r = (warp & 3) * 32 + lane, k = kb + r;
        const int tu = k < k_hi ? taps_used(k, f, n_ac) : 0;
        const int kmin = window_start(kb);
        const bool fits = (tu == n_ac && k - n_ac + 1 >= kmin) || k - tu + 1 == kmin;
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const int c0 = (warp >> 2) * 16 + part * 8;
          const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0;
          float G[tfir::kDigits][8];
#pragma unroll
          for (int m2 = 0; m2 < tfir::kDigits; ++m2) tfir::tmem_load8(at + kCols * m2, G[m2]);
          tfir::tmem_wait_loads();
          uint32_t bad = 0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float q = 1.0f / 512.0f;
            float e2, e1, e0;
            const float g3 = __fmaf_rn(G[4][c], q, G[3][c]);
            const float h2 = two_sum(G[2][c], __fmul_rn(g3, q), e2);
            const float h1 = two_sum(G[1][c], __fmul_rn(h2, q), e1);
            const float h0 = two_sum(G[0][c], __fmul_rn(h1, q), e0);
            const float lo = __fmaf_rn(__fmaf_rn(e2, q, e1), q, e0);
            const float res = __fadd_rn(h0, lo);
            const float rest = __fsub_rn(lo, __fsub_rn(res, h0));
            const float sl = S.slack[c0 + c];
            const float ac = __fmul_rn(res, S.unit[c0 + c]);
            const bool sure = __fadd_rn(res, __fadd_rn(rest, sl)) == res &&
                              __fadd_rn(res, __fsub_rn(rest, sl)) == res &&
                              (sl == 0.0f || fabsf(ac) > 1e-30f);
            AC[r * kPitch + c0 + c] = tu == 0 ? 0.0f : ac;
            if (tu > 0 && !(fits && sure)) bad |= 1u << c;
          }
          if (bad) {
            int p = atomicAdd(&S.listed, __popc(bad));
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (bad >> c & 1) list[p++] = (uint16_t)(r * kCols + c0 + c);
          }
        }
      }
      tfir::fence_before();
      sync_workers();
      const int listed = S.listed;
      for (int p = threadIdx.x; p < listed; p += kWorkers) {
        const int q = list[p], r = q / kCols, c = q - r * kCols;
        AC[r * kPitch + c] = dot2_row(vf + (int64_t)(kb + r) * 256 + c, TP,
                                      taps_used(kb + r, f, n_ac), n_ac, A.ac_sym != 0);
      }
      sync_workers();
      if (threadIdx.x == 0) S.listed = 0;
      // dS of the tile's rows
#pragma unroll 4
      for (int r = gw; r < k_hi - kb; r += 8) {
        const float xv = __ldg(vf + (int64_t)(kb + r) * 256 + sec);
        const float ms = __fmaf_rn(xv, A.scale, -AC[r * kPitch + sec]);
        DS[(n_dc + r) * kPitch + sec] = __fmul_rn(ms, ms);
      }
      sync_workers();
    }
    if (ok)
      finish_tile(t1 - 1);
    else if (threadIdx.x == 0)
      atomicOr(A.status, 1);
  }
  __syncthreads();
  if (warp == kIhcWarps) tfir::tmem_free(tmem);
}

size_t tensor_smem(int n_ac, int n_dc) {
  return 2 * (size_t)tfir::kHalfBytes + tfir::kTapBytes +
         ((size_t)n_dc + 2 * tfir::kRows) * kPitch * 4 + (size_t)n_ac * 4 + 16 +
         sizeof(TensorShared);
}

}  // namespace

bool ihc_tensor_fits(int n_ac, int n_dc) {
  return n_ac >= kTensorMinTaps && n_ac <= tfir::kMaxTaps &&
         tensor_smem(n_ac, n_dc) <= 227 * 1024;
}

int ihc_tensor_launch(const IHCArgs& A, const float* d_v, int n_runs, int exp_b, float slack,
                      cudaStream_t st) {
  const size_t smem = tensor_smem(A.n_ac, A.n_dc);
  CGB_TRY_CUDA(cudaFuncSetAttribute(ihc_tensor_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "cudaFuncSetAttribute(ihc tensor smem)");
  ihc_tensor_kernel<<<dim3((unsigned)n_runs, 256 / kCols), kThreads, smem, st>>>(A, d_v, exp_b,
                                                                                 slack);
  CGB_TRY_CUDA(cudaGetLastError(), "ihc_tensor_kernel launch");
  note_launch();
  return CGB_OK;
}

}  // namespace cgb
