// BM/OHC adaptive-step solver for few units: four warps per unit, for the
// calls that leave most of the chip idle with one warp per unit (bm_step.cu).
//
// What bounds such a call is one unit's chain of dependent operations: with a
// warp per unit a substep is ~2,300 warp instructions and ~7,600 cycles, on
// one scheduler, while 3 schedulers of the SM and most SMs have nothing to do.
// Here a unit is a CTA of four warps, one per scheduler, and a lane holds four
// sections of every state vector instead of eight.
//
// Split.  Warp w owns sections 64w .. 64w+63 and works on the window of 128
// sections 64w-32 .. 64w+95, lane m on 64w-32+4m .. +3 (own lanes: 8..23; the
// sections below 0 and above 255 have zero coefficients and stay zero).  The
// halo of 32 on each side is computed redundantly, bit for bit the values its
// owner has, so that a whole pressure solve of up to 32 Jacobi sweeps runs
// inside the warp: every sweep makes one more halo section on each side stale,
// and after the solve the halo's pressure comes from its owners through shared
// memory.  An outer iteration then has two block barriers (the velocity-error
// sums; the pressure with the acceleration maximum) instead of one per pair of
// sweeps: an exchange through shared memory costs ~50 cycles here, a shuffle
// 24, and a solve has 10 rounds.
//
// The three kinds of outer iteration are compiled apart, and the sums' shuffle
// rounds are spread over them; 1.4k warp instructions a substep, 3.4k cycles.
//
// Measured (GB300, 5 ms blocks with 1 ms overlap, kernel 17 / the default
// kernel's semantics), against a warp per unit: 1 unit 17.5 / 37.7 -> 10.0 /
// 22.2 ms, 152 units (one CTA per SM) 16.7 / 37.8 -> 9.2 / 21.7 ms, 304 units
// (two) 16.5 / 35.1 -> 11.9 / 25.4 ms.  Tried and slower: the next test's sums
// in the same exchange as the pressure (one barrier an iteration instead of
// two, 12.2 against 11.5 ms: its arithmetic is then ahead of the barrier),
// two-wide fmas in the two-step update (10.8 against 10.7), rounds of the sums
// replaced by wider reads of them (10.9 to 13.2), and the next iteration's
// predictor ahead of the step test's branch (11.9, with its right-hand side;
// 11.7 without): the moves cost more than the vote's latency.
//
// The arithmetic is run_unit's (bm_step.cu) operation for operation, so the
// results are the same bits; the sums over the sections keep its order.

#include <cuda_runtime.h>

#include <type_traits>

#include "bm_common.cuh"
#include "cgb_device.cuh"
#include "cgb_internal.h"

namespace cgb {
namespace {

constexpr int kQWarps = 4;
constexpr int kQThreads = kQWarps * 32;
constexpr int kQHalo = 32;  // sections of halo on each side of a warp's own 64
static_assert(kQuadMaxSweeps <= kQHalo, "a solve may not use up the halo");

// A lane's four sections as two pairs, seen from the neighbour that its pair 0
// faces: an even lane holds (s0, s1), (s2, s3), an odd lane (s3, s2), (s1, s0),
// s0 its lowest section.  Pair 0 then always faces the lane of the other parity
// on one side (lane - 1 of an even lane, lane + 1 of an odd one), pair 1 the
// lane ^ 1, and all lanes run the same code: along the lane
//   hA.x hA.y | r[0].x r[0].y r[1].x r[1].y | hB.x hB.y
// are consecutive sections, upwards in even lanes and downwards in odd ones.
__device__ __forceinline__ void lane_pairs(float4 q, bool odd, float2 (&r)[2]) {
  r[0] = odd ? f2(q.w, q.z) : f2(q.x, q.y);
  r[1] = odd ? f2(q.y, q.x) : f2(q.z, q.w);
}
__device__ __forceinline__ float4 lane_quad(const float2 (&r)[2], bool odd) {
  return odd ? make_float4(r[1].y, r[1].x, r[0].y, r[0].x)
             : make_float4(r[0].x, r[0].y, r[1].x, r[1].y);
}

// What the warps exchange in an outer iteration, twice (by iteration parity, so
// that one barrier per exchange is enough).  A lane's four values lie in the
// order that its pairs have; readers of a quad have its owner's parity.
struct __align__(16) QuadExchange {
  float4 p[80];      // pressure: lane m of warp w at 16 w + m; 8 zero quads at each end
  float4 dv[64];     // |dv| (reference order only)
  float2 sum[64];    // velocity error and margin of sections 4l .. 4l+3
  float ea[kQWarps]; // acceleration maxima of the warps' own sections
};

// REF: the reference schedule's sweep counts, known to the compiler.
template <int CTL, int ARITH, bool REF>
__global__ void __launch_bounds__(kQThreads, 2) bm_quad_kernel(const BMArgs A) {
  __shared__ QuadExchange S2[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool odd = lane & 1;
  const int base = 64 * warp - kQHalo + 4 * lane;  // lowest section
  const bool inside = base >= 0 && base < 256;
  const bool own = lane >= 8 && lane < 24;
  const bool sec0 = base == 0, sec255 = base == 252;
  // the lane pair 0 faces; outside the unit the lane itself: its zeros stay zeros
  // where the pressure at the ends is infinite
  const int pa = !inside ? lane : odd ? (lane + 1) & 31 : (lane + 31) & 31;
  const cgb_unit un = A.units[blockIdx.x];

  auto load_row = [&](const float* row, float outside, float2 (&r)[2]) {
    const float4 o = make_float4(outside, outside, outside, outside);
    lane_pairs(inside ? *reinterpret_cast<const float4*>(row + base) : o, odd, r);
  };
  float2 invM[2], rm[2], Rs[2], Ss[2], Qs[2], Stm[2], Rtm[2], gm[2], gs[2];
  load_row(A.secp + 0 * 256, 0.0f, invM);
  load_row(A.secp + 1 * 256, 0.0f, rm);
  load_row(A.secp + 2 * 256, 0.0f, Rs);
  load_row(A.secp + 3 * 256, 0.0f, Ss);
  load_row(A.secp + 4 * 256, 0.0f, Qs);
  load_row(A.secp + 5 * 256, 0.0f, gs);
  load_row(A.secp + 6 * 256, 0.0f, Stm);
  load_row(A.secp + 7 * 256, 1.0f, Rtm);  // 1: u = 0 / -1 outside, not 0 / 0
  {
    // gamma has no alignment rule: scalar loads
    const float* g = A.gamma + (int64_t)un.profile * 256;
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (inside) q = make_float4(g[base], g[base + 1], g[base + 2], g[base + 3]);
    lane_pairs(q, odd, gm);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) gs[k] = mul2(gm[k], gs[k]);
  // Two-step coefficients (bm_body of bm_step.cu): a_s on the lower second
  // neighbour, c_s on the upper one.  The term added first is the upper one in
  // sections with s mod 8 < 4 (even lanes), the lower one in the others.
  float2 K1[2], K2[2], KB[2];
  if (!ARITH) {
    float4 a4, b4, c4;
    float* pa4 = &a4.x;
    float* pb4 = &b4.x;
    float* pc4 = &c4.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int s = base + i;
      const float r = inside ? A.secp[256 + s] : 0.0f;
      const float rl = inside && s >= 1 ? A.secp[256 + s - 1] : 0.0f;
      const float ru = inside && s <= 254 ? A.secp[256 + s + 1] : 0.0f;
      pa4[i] = (s >= 2 && s <= 253) ? __fmul_rn(r, rl) : 0.0f;
      pc4[i] = s <= 253 ? __fmul_rn(r, ru) : 0.0f;
      pb4[i] =
          __fmul_rn(r, __fadd_rn((s >= 1 && s <= 253) ? rl : 0.0f, s <= 252 ? ru : 0.0f));
    }
    lane_pairs(odd ? a4 : c4, odd, K1);
    lane_pairs(odd ? c4 : a4, odd, K2);
    lane_pairs(b4, odd, KB);
  }
  // section 255 (pair 0's x of its lane) has coefficient 0, section 254 (its y)
  // no lower neighbour
  if (sec255) rm[0].x = 0.0f;
  const float lo = sec255 ? 0.0f : 1.0f;
  // 1/m of the two sections next to the lane
  const float2 rmh = f2(__shfl_sync(kFull, rm[0].x, pa), __shfl_xor_sync(kFull, rm[1].y, 1));

  float2 x0[2], v0[2], a0[2], y0[2], u0[2], ps0[2], dp0[2];
  float2 x[2], v[2], a[2], y[2], u[2], ps[2], dp[2], p[2], Yrm[2], G[2], Ptm[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    x0[k] = v0[k] = a0[k] = y0[k] = u0[k] = ps0[k] = dp0[k] = f2b(0.0f);
    x[k] = v[k] = a[k] = y[k] = u[k] = ps[k] = dp[k] = f2b(0.0f);
    p[k] = Yrm[k] = G[k] = Ptm[k] = f2b(0.0f);
  }
  float w0 = 0.f, wd0 = 0.f, wdd0 = 0.f, w = 0.f, wd = 0.f, wdd = 0.f;

  const float mtt = un.mtt, mmspt = un.mmspt;
  const float* inb = A.in + un.in_base;
  float* outb = A.out + un.out_base * 256;
  int32_t* fb = A.failed ? A.failed + un.out_base : nullptr;
  float* cb = A.conv ? A.conv + un.out_base * 3 : nullptr;
  float dt = A.dt0, tau_f = 0.0f;
  int n = un.start;
  // input samples n, n + 1 and, loaded a sample ahead, n + 2 (the last sample
  // that a unit uses is end + 1)
  float sx0 = inb[n], sx1 = inb[n + 1], sx2 = inb[min(n + 2, un.end + 1)];
  int fail_flag = 0;
  long long n_sub = 0, n_it = 0, n_sw = 0;
  int n_failed = 0, n_written = 0, status = 0, sub_in_sample = 0;
  float smp_dt = 0.0f, smp_sub = 0.0f, smp_it = 0.0f;
  // this lane's places in the exchange: its own quad, the values it adds up
  const int quad = 16 * warp + lane;
  // BMOHC_NEW_kernel's tree reads section lane + 32 k: quads of odd lanes lie
  // from their highest section down
  const int dv_at = lane ^ ((lane & 4) ? 3 : 0);
  if (threadIdx.x < 8) {
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    S2[0].p[threadIdx.x] = S2[1].p[threadIdx.x] = z;
    S2[0].p[72 + threadIdx.x] = S2[1].p[72 + threadIdx.x] = z;
  }
  int buf = 0;

  // the pair sums p_{s-1} + p_{s+1} along the lane, h1 / h2 the two sections
  // next to it
  auto neighbours = [&](const float2 (&q)[2], float h1, float h2, float2 (&T)[2]) {
    if (ARITH) {  // without the lower neighbours of 254 and 255, also where they are not finite
      T[0] = f2(sec255 ? 0.0f : __fadd_rn(h1, q[0].y),
                sec255 ? q[0].x : __fadd_rn(q[1].x, q[0].x));
    } else {
      T[0] = f2(__fadd_rn(h1, q[0].y), __fmaf_rn(lo, q[1].x, q[0].x));
    }
    T[1] = f2(__fadd_rn(q[0].y, q[1].y), __fadd_rn(q[1].x, h2));
  };
  auto sweep = [&](float2 T, float2 r, float2 Y) {
    return ARITH ? mul2(sub2(Y, T), r) : fma2(neg2(T), r, Y);
  };

  while (n < un.end) {
    if (++sub_in_sample > A.max_sub) {
      status = 1;
      break;
    }
    // known before the step, so that their latency passes under it
    const bool emit = __all_sync(kFull, tau_f > A.tout_f);
    // (n is the same in all lanes; the vote that tells the compiler so pays in the own
    // order, 10.0 against 10.2 ms, and costs in the reference's, 22.6 against 22.2)
    const bool owned_row = ARITH ? n >= un.out_first : __all_sync(kFull, n >= un.out_first);
    const float delta = __fmul_rn(tau_f, A.fs_f);
    const float smp = __fmaf_rn(sx1, delta, __fmul_rn(sx0, __fsub_rn(1.0f, delta)));
    const float hdt = __fmul_rn(dt, 0.5f);
    const float2 dt2 = f2b(dt), hdt2 = f2b(hdt);

    // One outer iteration; true to go on.  The three kinds an iteration can be
    // are compiled separately, each as straight-line code around its solve, so
    // that the sums' shuffle chains pass under the TM update and the sweeps:
    //   FIRST  the first of a step: the Euler predictor (the trapezoid rule on
    //          the previous derivatives twice), no step test
    //   SLOW   the first two: the TM update and jslow sweeps
    auto iterate = [&](auto first_c, auto slow_c) -> bool {
      constexpr bool FIRST = decltype(first_c)::value, SLOW = decltype(slow_c)::value;
      buf ^= 1;
      QuadExchange& S = S2[buf];
      // the pressure next to the lane, for the first round of the solve: it
      // is known since the iteration before
      const float2 pA = f2(__shfl_sync(kFull, p[0].y, pa), __shfl_sync(kFull, p[0].x, pa));
      const float2 pB = f2(__shfl_xor_sync(kFull, p[1].y, 1), __shfl_xor_sync(kFull, p[1].x, 1));
      float2 dv[2], fl[2];
      const float2 mtt2 = f2b(mtt);
      bool fault = false;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float2 vn = fma2(add2(a0[k], FIRST ? a0[k] : a[k]), hdt2, v0[k]);
        if (!FIRST) {
          dv[k] = abs2(sub2(vn, v[k]));
          const float2 thr = max2(mtt2, mul2(vn, dt2));
          if (CTL == 0) fl[k] = sub2(dv[k], thr);
          else fault = fault || dv[k].x > thr.x || dv[k].y > thr.y;
        }
        v[k] = vn;
        x[k] = fma2(add2(v0[k], vn), hdt2, x0[k]);
        y[k] = fma2(add2(u0[k], FIRST ? u0[k] : u[k]), hdt2, y0[k]);
        ps[k] = fma2(add2(dp0[k], FIRST ? dp0[k] : dp[k]), hdt2, ps0[k]);
      }
      w = __fmaf_rn(__fadd_rn(wd0, FIRST ? wd0 : wd), hdt, w0);
      wd = __fmaf_rn(__fadd_rn(wdd0, FIRST ? wdd0 : wdd), hdt, wd0);
      // OHC / TM coupling, G and the right-hand side Y
      if (SLOW) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float2 d = sub2(y[k], x[k]);
          const float2 Pohc = mul2(gs[k], d);
          const float2 targ = mul2(f2b(A.ratio), ps[k]);
          const float2 t = ARITH ? tanhf2(targ) : own_tanhf2(targ);
          const float2 dL = mul2(f2b(A.nas), t);
          const float2 Aa = mul2(f2b(A.al), fma2(t, t, f2b(-1.0f)));
          const float2 N1 =
              ARITH ? fma2(f2b(A.e2), v[k], fma2(f2b(A.e1), d, mul2(f2b(A.nw), ps[k])))
                    : fma2(f2b(A.e1), d, fma2(f2b(A.e2), v[k], mul2(f2b(A.nw), ps[k])));
          const float2 N = fma2(Stm[k], dL, mul2(mul2(N1, Rtm[k]), Aa));
          const float2 Pp = fma2(Stm[k], y[k], Pohc);
          const float2 num = fma2(neg2(gm[k]), N, Pp);
          const float2 den = mul2(Rtm[k], fma2(mul2(gm[k], Aa), f2b(A.e2), f2b(-1.0f)));
          if (ARITH) {
            u[k] = fdividef2(num, den);
          } else {
            const float2 q = mul2(num, own_rcpf2(abs2(den)));
            u[k] = f2(den.x < 0.0f ? -q.x : q.x, den.y < 0.0f ? -q.y : q.y);
          }
          Ptm[k] = fma2(Rtm[k], u[k], mul2(Stm[k], y[k]));
        }
      }
      float Y0;  // section 0
      if (ARITH)
        Y0 = __fmul_rn(A.dxa0, __fmaf_rn(A.gme, smp, __fmaf_rn(A.na1, w, __fmul_rn(A.na2, wd))));
      else
        Y0 = __fmul_rn(A.dxa0, __fmaf_rn(A.na1, w, __fmaf_rn(A.na2, wd, __fmul_rn(A.gme, smp))));
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        float2 g = mul2(Rs[k], fma2(f2b(A.ar), mul2(v[k], v[k]), f2b(1.0f)));
        g = fma2(g, v[k], mul2(Ss[k], x[k]));
        G[k] = sub2(neg2(g), Ptm[k]);
        float2 Yk = mul2(mul2(f2b(A.dx2), G[k]), Qs[k]);
        if (k == 0) Yk.x = sec0 ? Y0 : (sec255 ? 0.0f : Yk.x);
        Yrm[k] = ARITH ? Yk : mul2(Yk, rm[k]);
      }

      // Jacobi sweeps inside the warp's window
      const int J = REF ? (SLOW ? kSlowSweeps : kFastSweeps) : (SLOW ? A.jslow : A.jfast);
      const float2 Yrmh =
          f2(__shfl_sync(kFull, Yrm[0].x, pa), __shfl_xor_sync(kFull, Yrm[1].y, 1));
      // Velocity error and margin: the lanes' sums of four sections go to
      // shared memory, and every warp adds the 64 of them in the order of the
      // butterfly over a whole warp of eight sections a lane.  Each round is
      // a shuffle (24 cycles) and an addition that nothing needs before the
      // step test: the five rounds are spread over the iteration, one between
      // two other shuffles or barriers each, where other work fills their
      // latency.  (Next to each other in front of the solve they held it up:
      // the warp issues in order.  11.2 / 23.4 -> 10.7 / 22.6 ms.)
      float2 sum = f2b(0.0f), sum_t;
      bool faulty = false;
      auto round = [&](int o) {
        sum_t = f2(__shfl_xor_sync(kFull, sum.x, o),
                   CTL == 0 ? __shfl_xor_sync(kFull, sum.y, o) : 0.0f);
        sum = add2(sum, sum_t);
      };
      // the places of a fast iteration in turn: between its two sweeps, after
      // them, before and after the acceleration maximum, after the barrier
      auto place = [&](int k) {
        if (FIRST || SLOW) return;
        if (k == 1) round(16);
        if (k == (ARITH ? 1 : 2)) round(8);
        if (k == (ARITH ? 2 : 3)) round(4);
        if (k == (ARITH ? 3 : 4)) round(2);
        if (k == (ARITH ? 4 : 5)) round(1);
      };
      if (!FIRST) {
        if (ARITH) {
          if (own) S.dv[quad - 8] = make_float4(dv[0].x, dv[0].y, dv[1].x, dv[1].y);
        } else {
          float2 q = f2b(__fadd_rn(__fadd_rn(dv[0].x, dv[0].y), __fadd_rn(dv[1].x, dv[1].y)));
          if (CTL == 0)
            q.y = __fadd_rn(__fadd_rn(fl[0].x, fl[0].y), __fadd_rn(fl[1].x, fl[1].y));
          if (own) S.sum[quad - 8] = q;
        }
        if (CTL == 1)
          faulty = __syncthreads_or(own && fault) != 0;
        else
          __syncthreads();
        if (ARITH) {
          // BMOHC_NEW_kernel's tree (ref_tree_sum of bm_step.cu)
          float e[8];
#pragma unroll
          for (int k = 0; k < 8; ++k)
            e[k] = reinterpret_cast<const float*>(S.dv)[dv_at + 32 * k];
#pragma unroll
          for (int t = 4; t >= 1; t >>= 1)
#pragma unroll
            for (int k = 0; k < t; ++k) e[k] = __fadd_rn(e[k], e[k + t]);
          sum.x = e[0];
        } else {
          const float4 q = *reinterpret_cast<const float4*>(&S.sum[2 * lane]);
          sum = f2(__fadd_rn(q.x, q.z), __fadd_rn(q.y, q.w));
        }
      }

      // two sweeps with one shuffle round: the first also on the two sections
      // next to the lane
      auto sweep_pair = [&](float2 hA, float2 hB, bool only) {
        float2 T[2], q[2];
        const float2 Th = f2(__fadd_rn(hA.x, p[0].x), __fadd_rn(p[1].y, hB.y));
        const float2 qh = sweep(Th, rmh, Yrmh);
        neighbours(p, hA.y, hB.x, T);
        q[0] = sweep(T[0], rm[0], Yrm[0]);
        q[1] = sweep(T[1], rm[1], Yrm[1]);
        if (only) place(1);
        neighbours(q, qh.x, qh.y, T);
        p[0] = sweep(T[0], rm[0], Yrm[0]);
        p[1] = sweep(T[1], rm[1], Yrm[1]);
      };
      float2 C2[2];
      auto two_step_setup = [&]() {
        float2 T[2];
        neighbours(Yrm, Yrmh.x, Yrmh.y, T);
        C2[0] = fma2(neg2(T[0]), rm[0], Yrm[0]);
        C2[1] = fma2(neg2(T[1]), rm[1], Yrm[1]);
      };
      // two sweeps as one update over the second neighbours (bm_step.cu)
      auto two_step = [&](float2 hA, float2 hB) {
        // (scalar: an fma on three pairs of registers takes 3 cycles, two fmas 2.4)
        auto f2s = [](float2 a, float2 b, float2 c) {
          return f2(__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y));
        };
        const float2 r0 = f2s(K2[0], hA, f2s(K1[0], p[1], f2s(KB[0], p[0], C2[0])));
        const float2 r1 = f2s(K2[1], p[0], f2s(K1[1], hB, f2s(KB[1], p[1], C2[1])));
        p[0] = r0;
        p[1] = r1;
      };
      auto halo = [&](float2& hA, float2& hB) {
        hA = f2(__shfl_sync(kFull, p[0].y, pa), __shfl_sync(kFull, p[0].x, pa));
        hB = f2(__shfl_xor_sync(kFull, p[1].y, 1), __shfl_xor_sync(kFull, p[1].x, 1));
      };
      const bool unrolled = SLOW && !ARITH && J == kSlowSweeps;
      if (!FIRST && SLOW && !unrolled) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) round(o);
      }
      float2 hA = pA, hB = pB;
      int it = 0;
      if (unrolled) {  // the reference schedule's slow count
        two_step_setup();
        two_step(hA, hB);
#pragma unroll
        for (int r = 1; r < kSlowSweeps / 2; ++r) {
          halo(hA, hB);
          if (!FIRST && r <= 5) round(32 >> r);
          two_step(hA, hB);
        }
        it = kSlowSweeps;
      } else if (!SLOW && J == kFastSweeps) {  // and its fast count
        sweep_pair(hA, hB, true);
        it = kFastSweeps;
      } else if (!ARITH && J >= 4) {
        place(1);
        two_step_setup();
        for (; it + 1 < J; it += 2) {
          two_step(hA, hB);
          halo(hA, hB);
        }
      } else {
        place(1);
        for (; it + 1 < J; it += 2) {
          sweep_pair(hA, hB, false);
          halo(hA, hB);
        }
      }
      if (it < J) {  // an odd count ends with one plain sweep
        float2 T[2];
        neighbours(p, hA.y, hB.x, T);
        p[0] = sweep(T[0], rm[0], Yrm[0]);
        p[1] = sweep(T[1], rm[1], Yrm[1]);
      }
      n_sw += J;
      place(2);

      // The pressure of the own sections and their acceleration maximum go to
      // shared memory together: one barrier, after which the halo takes its
      // owners' pressure.
      if (own) S.p[quad] = make_float4(p[0].x, p[0].y, p[1].x, p[1].y);
      if (!FIRST) {
        float eap = 0.0f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float2 da = abs2(sub2(a[k], mul2(add2(p[k], G[k]), invM[k])));
          eap = fmaxf(eap, fmaxf(da.x, da.y));
        }
        place(3);
        const float eaw = warp_max_xor(own ? eap : 0.0f);
        if (lane == 0) S.ea[warp] = eaw;
      }
      place(4);
      __syncthreads();
      const float4 em = *reinterpret_cast<const float4*>(S.ea);
      const float p0 = S.p[8].x;  // section 0
      const float4 pq = S.p[quad];
      place(5);

      // Step test: the decision is voted on, which makes it uniform for the
      // compiler, before the rest of the iteration, which covers the vote.
      bool go_on = true;
      if (!FIRST) {
        const float ev = sum.x;
        if (CTL == 0) faulty = sum.y > 0.0f;
        const float ea = fmaxf(fmaxf(em.x, em.y), fmaxf(em.z, em.w));
        const float num = __fmul_rn(ea, dt);
        const bool lcheck = ev > mmspt;
        const float L = lcheck && ARITH ? __fdividef(num, ev) : 0.0f;
        const bool l_big = ARITH ? L > 6.0f : lcheck && num > __fmul_rn(6.0f, ev);
        const bool l_small = ARITH ? L < 0.5f : !lcheck || num < __fmul_rn(0.5f, ev);
        const bool grow = !l_big && !faulty && l_small;
        const float up = __fmul_rn(dt, 2.0f), down = __fmul_rn(dt, 0.5f);
        dt = l_big ? (down < A.dtmin ? A.dtmin : down)
                   : (grow ? (up > A.dtmax ? A.dtmax : up) : dt);
        go_on = __all_sync(kFull, !l_big && !grow);
      }
      p[0] = f2(pq.x, pq.y);
      p[1] = f2(pq.z, pq.w);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        a[k] = mul2(add2(p[k], G[k]), invM[k]);
        const float2 d = sub2(y[k], x[k]);
        if (ARITH)
          dp[k] = fma2(f2b(A.nw), ps[k],
                       fma2(f2b(A.e1), d, mul2(f2b(A.e2), sub2(u[k], v[k]))));
        else
          dp[k] = fma2(f2b(A.e1), d,
                       fma2(f2b(A.e2), sub2(u[k], v[k]), mul2(f2b(A.nw), ps[k])));
      }
      if (ARITH) {
        wdd = __fmul_rn(A.rsow, __fadd_rn(__fmaf_rn(A.na2, wd, __fmul_rn(A.na1, w)),
                                          __fmaf_rn(A.gme, smp, p0)));
      } else {
        const float ws = __fmaf_rn(A.na1, w, __fmaf_rn(A.na2, wd, __fmaf_rn(A.gme, smp, p0)));
        wdd = A.ow_pow2 ? __fmul_rn(ws, A.rsow) : __fdiv_rn(ws, A.sow);
      }
      return go_on;
    };

    using Yes = std::true_type;
    using No = std::false_type;
    int out_loop = 1;
    iterate(Yes(), Yes());
    bool another = true;
    if (A.max_outer > 1) {
      another = iterate(No(), Yes());
      ++out_loop;
      while (another && out_loop < A.max_outer) {
        another = iterate(No(), No());
        ++out_loop;
      }
    }
    // a step that reaches max_outer iterations counts as failed, also where
    // the last of them passes the test
    if (out_loop >= A.max_outer) fail_flag = 1;
    ++n_sub;
    n_it += out_loop;
    smp_sub = __fadd_rn(smp_sub, 1.0f);
    smp_dt = __fadd_rn(smp_dt, dt);
    smp_it = __fadd_rn(smp_it, (float)out_loop);

    if (emit) {
      tau_f = __fsub_rn(tau_f, A.tout_f);
      sx0 = sx1;
      sx1 = sx2;
      sx2 = inb[min(n + 3, un.end + 1)];
      if (owned_row) {
        if (own) {
          float* row = outb + (int64_t)n * 256 + base;
          *reinterpret_cast<float4*>(row) = lane_quad(v, odd);
          if (A.host_delta)
            *reinterpret_cast<float4*>(reinterpret_cast<char*>(row) + A.host_delta) =
                lane_quad(v, odd);
        }
        if (threadIdx.x == 0) {
          if (fb) fb[n] = fail_flag;
          if (cb) {
            cb[(int64_t)n * 3 + 0] = __fdiv_rn(smp_dt, smp_sub);
            cb[(int64_t)n * 3 + 1] = smp_sub;
            cb[(int64_t)n * 3 + 2] = __fdiv_rn(smp_it, smp_sub);
          }
        }
        ++n_written;
        n_failed += fail_flag;
      }
      fail_flag = 0;
      sub_in_sample = 0;
      smp_dt = smp_sub = smp_it = 0.0f;
      ++n;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      x0[k] = x[k];
      v0[k] = v[k];
      a0[k] = a[k];
      y0[k] = y[k];
      u0[k] = u[k];
      ps0[k] = ps[k];
      dp0[k] = dp[k];
    }
    w0 = w;
    wd0 = wd;
    wdd0 = wdd;
    tau_f = __fadd_rn(tau_f, dt);
  }
  if (A.stats && threadIdx.x == 0) {
    cgb_unit_stats* st = A.stats + blockIdx.x;
    st->substeps = n_sub;
    st->iterations = n_it;
    st->sweeps = n_sw;
    st->failed_samples = n_failed;
    st->written_samples = n_written;
    st->status = status;
  }
}

}  // namespace

int bm_quad_launch(const BMArgs& A, int controller, int arith, cudaStream_t st) {
  const unsigned grid = (unsigned)A.n_units;
  // The reference schedule's sweep counts compiled in: 1 unit 10.7 -> 10.0 ms
  // (kernel 17); no gain for the reference's order.
  const bool schedule = A.jslow == kSlowSweeps && A.jfast == kFastSweeps;
  if (arith)
    bm_quad_kernel<1, 1, false><<<grid, kQThreads, 0, st>>>(A);
  else if (controller == 1 && schedule)
    bm_quad_kernel<1, 0, true><<<grid, kQThreads, 0, st>>>(A);
  else if (controller == 1)
    bm_quad_kernel<1, 0, false><<<grid, kQThreads, 0, st>>>(A);
  else if (schedule)
    bm_quad_kernel<0, 0, true><<<grid, kQThreads, 0, st>>>(A);
  else
    bm_quad_kernel<0, 0, false><<<grid, kQThreads, 0, st>>>(A);
  CGB_TRY_CUDA(cudaGetLastError(), "bm_quad_kernel launch");
  note_launch();
  return CGB_OK;
}

}  // namespace cgb
