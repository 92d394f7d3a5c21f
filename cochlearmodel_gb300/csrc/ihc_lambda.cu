// Fused IHC + auditory-nerve rate (lambda) kernel: reference RunIHCKernel
// (src/cochlea.cu:3573-3644) = CudaUnifiedCalcIHC (:3431-3506) followed by
// CudaCalcLambda (:3365-3408), with the decoupled FIR look-back rule of
// DeviceCudaFIRFilter (:2712-2730).
//
// Per point (t, s) of a frame:
//   AC  = sum_{i<tu(t)} b_i v[t-i]          (AC low-pass, taps pre-scaled)
//   dS  = (scale v - AC)^2
//   DC  = sum_{i<tu(t)} d_i dS[t-i]         (DC moving average)
//         with uniform taps d (the reference's DC filter): d * S(t), S the
//         window sum, re-summed at every 32nd frame row (and where the
//         look-back rule restarts the window) and otherwise updated by
//         adding dS[t] and removing dS[t-tu]; all in compensated (TwoSum)
//         arithmetic
//   IHC = log10(max(10^ihc_s (eta_AC AC + eta_DC DC), 0) + 1e-20)
//   lambda_j = s ? min(SAT, max(A_js IHC, spont_j)) : spont_j,  j = 0..2
// in FP32, each FIR accumulated with a compensated dot product (Dot2).
//
// This file holds the FP32 kernel, the host side of the stage and the IIR form of the
// AC filter.  The same stage with the AC filter on the tensor cores is ihc_tensor.cu;
// ihc_lambda_impl gives it the calls that it is built for (64 to 257 taps whose digit
// sums it holds, a uniform DC filter, no debug stage, no AC given) where the frame
// table makes it the faster one (tensor_faster).
//
// The FP32 kernel: one CTA = 32 sections x a run of consecutive TR-row tiles.
// Each tile's velocity window (TR rows plus the look-back) is staged into
// shared memory by TMA (cp.async.bulk.tensor.2d, 64-row boxes, completion on
// an mbarrier with a bounded wait), the next tile's while the current one
// finishes; AC and dS are computed from shared memory with 8-row register
// blocking, then DC, IHC and lambda, and the three lambda planes are written
// with coalesced 128-byte rows.

#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <atomic>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "ihc_common.cuh"
#include "ihc_tensor.h"

namespace cgb {
namespace {

constexpr int kBoxRows = 64;   // rows per TMA box
constexpr int kRB = 8;         // output rows per register block
constexpr int kTilesPerRun = 8;  // consecutive tiles per CTA (short runs)

// Test-only fault injection (cgb_ihc_set_fault_injection): the next launches
// arm the first staging mbarrier without issuing its copies (the tensor kernel
// leaves out its first products), so the bounded wait runs out and the kernel
// reports status bit 1.
int g_fault_skip_copy = 0;

// FIR of one 8-row block, rows kb..kb+7 all using `taps` taps.  src points at
// the staged row of output kb (lane's column); rows above it are older.  One
// shared-memory load feeds the eight rows' accumulators.  Rows r and r+4 form
// pair r, so the per-tap shift of the window moves whole pairs and only pair
// 0 is assembled from the newly loaded row.  The last step loads one row
// beyond the oldest tap (unused; the caller stages it).
__device__ __forceinline__ void fir_block8(const float* __restrict__ src,
                                           const float* __restrict__ b, int taps,
                                           float (&out)[kRB]) {
  float2 W[4];
  Dot2x2 acc[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    acc[j].init();
    W[j] = f2(src[j * kSecTile], src[(j + 4) * kSecTile]);
  }
#pragma unroll 4
  for (int i = 0; i < taps; ++i) {
    const float2 bi = f2b(b[i]);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j].add(bi, W[j]);
    const float w3 = W[3].x;
    W[3] = W[2];
    W[2] = W[1];
    W[1] = W[0];
    W[0] = f2(src[-(i + 1) * kSecTile], w3);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 r = acc[j].result();
    out[j] = r.x;
    out[j + 4] = r.y;
  }
}

// fir_block8 for a symmetric (linear-phase) filter of n taps, b_k = b_{n-1-k}:
// for each tap pair k the rows t-k and t-(n-1)+k are added exactly first
// (Dot2::add_pair), then the centre tap of an odd filter.  Two windows move
// in opposite directions: W1 (rows t-k, as in fir_block8) and W2 (rows
// t-(n-1)+k), one shared-memory load each per tap pair.  The rows read lie
// in [kb - n + 1, kb + 7], inside the staged window.
__device__ __forceinline__ void fir_block8_sym(const float* __restrict__ src,
                                               const float* __restrict__ b, int n,
                                               float (&out)[kRB]) {
  float2 W1[4], W2[4];
  Dot2x2 acc[4];
  const int o2 = -(n - 1) * kSecTile;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    acc[j].init();
    W1[j] = f2(src[j * kSecTile], src[(j + 4) * kSecTile]);
    W2[j] = f2(src[o2 + j * kSecTile], src[o2 + (j + 4) * kSecTile]);
  }
  const int half = n / 2;
#pragma unroll 2
  for (int k = 0; k < half; ++k) {
    const float2 bk = f2b(b[k]);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j].add_pair(bk, W1[j], W2[j]);
    const float w13 = W1[3].x;
    W1[3] = W1[2];
    W1[2] = W1[1];
    W1[1] = W1[0];
    W1[0] = f2(src[-(k + 1) * kSecTile], w13);
    const float w20 = W2[0].y;
    W2[0] = W2[1];
    W2[1] = W2[2];
    W2[2] = W2[3];
    W2[3] = f2(w20, src[o2 + (k + 8) * kSecTile]);
  }
  if (n & 1) {
    const float2 bc = f2b(b[half]);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j].add(bc, W1[j]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 r = acc[j].result();
    out[j] = r.x;
    out[j + 4] = r.y;
  }
}

// One row of a symmetric filter with all n taps (the order of fir_block8_sym).
__device__ __forceinline__ float fir_row_sym(const float* __restrict__ src,
                                             const float* __restrict__ b, int n) {
  Dot2 acc;
  acc.init();
  for (int k = 0; k < n / 2; ++k) acc.add_pair(b[k], src[-k * kSecTile], src[-(n - 1 - k) * kSecTile]);
  if (n & 1) acc.add(b[n / 2], src[-(n / 2) * kSecTile]);
  return acc.result();
}

__device__ __forceinline__ float fir_row(const float* __restrict__ src,
                                         const float* __restrict__ b, int tu) {
  Dot2 acc;
  acc.init();
  for (int i = 0; i < tu; ++i) acc.add(b[i], src[-i * kSecTile]);
  return acc.result();
}

// Stages velocity rows [y0, y0 + boxes * 64) of sections s0..s0+31 into X
// (TMA, completion on mbar).  Called by one thread after a block barrier that
// ends all reads of X; the proxy fence orders those generic-proxy reads
// before the asynchronous writes.
__device__ __forceinline__ void stage_rows(const CUtensorMap* vmap, float* X, uint64_t* mbar,
                                           int boxes, int y0, int s0, bool skip = false) {
  const uint32_t bytes = (uint32_t)boxes * kBoxRows * kSecTile * 4;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)),
               "r"(bytes)
               : "memory");
  if (skip) return;  // test-only: the transaction count is never met
  for (int bxi = 0; bxi < boxes; ++bxi) {
    const int y = y0 + bxi * kBoxRows;  // may be negative or past the end: zero fill
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(X + (size_t)bxi * kBoxRows * kSecTile)),
        "l"(vmap), "r"(s0), "r"(y), "r"(smem_u32(mbar))
        : "memory");
  }
}

// One CTA = 32 sections x a run of up to A.run consecutive tiles of TR rows
// of one frame, processed in order.  The first tile of the run computes AC
// and dS on the DC filter's look-back rows as well; later tiles inherit those
// n_dc - 1 rows of dS from the previous tile (shifted down in shared memory)
// and stage only the AC filter's look-back (plus one row), the next tile's rows being copied
// by TMA while the current tile's DC/IHC/lambda phase runs.
__global__ void __launch_bounds__(kIhcWarps * 32)
    ihc_lambda_kernel(const __grid_constant__ CUtensorMap vmap, const IHCArgs A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  // layout: X [xrows][32] | dS [TR + n_dc][32] | AC [TR][32] | taps | mbarrier
  float* X = reinterpret_cast<float*>(smem_raw);
  float* DS = X + (size_t)A.xrows * kSecTile;
  float* ACb = DS + (size_t)(A.TR + A.n_dc) * kSecTile;
  float* TP = ACb + (size_t)A.TR * kSecTile;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(
      (reinterpret_cast<uintptr_t>(TP + A.n_ac + A.n_dc) + 15) & ~uintptr_t(15));

  // locate the frame and the run
  const int bx = blockIdx.x;
  int lo = 0, hi = A.n_frames;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (A.tile_prefix[mid] <= bx) lo = mid; else hi = mid;
  }
  const cgb_ihc_frame f = A.frames[lo];
  const int tiles = (f.lam_rows + A.TR - 1) / A.TR;
  const int t0 = (bx - A.tile_prefix[lo]) * A.run;
  const int t1 = min(t0 + A.run, tiles);
  const int s0 = blockIdx.y * kSecTile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int boxes_first = A.xrows / kBoxRows;
  // later tiles stage rows from row0 - n_ac: the register-blocked FIR loads
  // one row beyond its oldest tap on its last step (a value it never uses),
  // and that row must lie inside the staged window
  const int boxes_next = (A.TR + A.n_ac + kBoxRows - 1) / kBoxRows;

  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  for (int i = threadIdx.x; i < A.n_ac + A.n_dc; i += blockDim.x) TP[i] = A.taps[i];
  __syncthreads();
  // staged rows of the first tile start one row below the oldest row either
  // filter reads; those of later tiles below the oldest row the AC filter reads
  if (threadIdx.x == 0)
    stage_rows(&vmap, X, mbar, boxes_first, (int)f.v_row0 + t0 * A.TR - A.n_ac - A.n_dc + 1, s0,
               A.skip_first_copy != 0);

  const float* bac = TP;
  const float* bdc = TP + A.n_ac;
  const float scale = A.scale;
  const int s = s0 + lane;
  const float dmg = A.dmg[(size_t)f.ihc_profile * 256 + s];
  const float a0 = A.aihc[0 * 256 + s], a1 = A.aihc[1 * 256 + s], a2 = A.aihc[2 * 256 + s];
  const bool sec0 = s == 0;

  for (int t = t0; t < t1; ++t) {
    const bool first = t == t0;
    const int row0 = t * A.TR;
    const int TRt = min(A.TR, f.lam_rows - row0);
    const int xbase = first ? row0 - A.n_ac - A.n_dc + 1 : row0 - A.n_ac;
    const int dsbase = row0 - A.n_dc;
    if (!wait_stage(mbar, (uint32_t)((t - t0) & 1))) {
      if (threadIdx.x == 0) atomicOr(A.status, 1);
      return;
    }
    if (!first) {
      // dS of rows row0 - n_dc + 1 .. row0 - 1 from the previous tile's buffer
      for (int i = 1 + warp; i < A.n_dc; i += kIhcWarps)
        DS[(size_t)i * kSecTile + lane] = DS[(size_t)(i + A.TR) * kSecTile + lane];
      __syncthreads();
    }

    // phase 1: AC and dS on rows [k_lo, row0 + TRt)
    const int k_lo = first ? max(0, row0 - A.n_dc + 1) : row0, k_hi = row0 + TRt;
    for (int kb = k_lo + warp * kRB; kb < k_hi; kb += kIhcWarps * kRB) {
      const int nr = min(kRB, k_hi - kb);
      bool fast = nr == kRB;
#pragma unroll
      for (int r = 0; r < kRB; ++r)
        fast = fast && taps_used(kb + r, f, A.n_ac) == A.n_ac;
      float acc[kRB];
      const float* src = X + (size_t)(kb - xbase) * kSecTile + lane;
      if (A.ac_ext) {
#pragma unroll
        for (int r = 0; r < kRB; ++r)
          acc[r] = r < nr ? A.ac_ext[((int64_t)f.v_row0 + kb + r) * 256 + s] : 0.0f;
      } else if (fast) {
        if (A.ac_sym)
          fir_block8_sym(src, bac, A.n_ac, acc);
        else
          fir_block8(src, bac, A.n_ac, acc);
      } else {
#pragma unroll
        for (int r = 0; r < kRB; ++r) {
          const int tu = taps_used(kb + r, f, A.n_ac);
          acc[r] = r >= nr ? 0.0f
                   : (A.ac_sym && tu == A.n_ac ? fir_row_sym(src + r * kSecTile, bac, tu)
                                               : fir_row(src + r * kSecTile, bac, tu));
        }
      }
#pragma unroll
      for (int r = 0; r < kRB; ++r) {
        if (r < nr) {
          const int k = kb + r;
          const float ms = __fmaf_rn(src[r * kSecTile], scale, -acc[r]);
          const float ds = __fmul_rn(ms, ms);
          DS[(size_t)(k - dsbase) * kSecTile + lane] = ds;
          if (k >= row0) {
            ACb[(size_t)(k - row0) * kSecTile + lane] = acc[r];
            if (A.stage == 9 || A.stage == 11)
              A.stage_out[((int64_t)f.lam_row0 + k) * 256 + s] = A.stage == 9 ? acc[r] : ds;
          }
        }
      }
    }
    __syncthreads();
    // X is free: stage the next tile while this one finishes
    if (threadIdx.x == 0 && t + 1 < t1)
      stage_rows(&vmap, X, mbar, boxes_next, (int)f.v_row0 + (t + 1) * A.TR - A.n_ac, s0);

    // phase 2: DC, IHC and lambda on rows [row0, row0 + TRt).  Pass 1
    // computes each row's pre-synaptic value eta_AC * AC + eta_DC * DC and
    // leaves it in the row's ACb slot.  Pass 2 turns pre-synaptic values into
    // IHC and lambda, kEmitRows rows per warp at a time: their arithmetic is
    // branch-free and independent, so the rows' dependent chains (log10)
    // interleave; the stores follow, behind the uniform output branches.
    auto set_pre = [&](int k, float dc) {
      float& slot = ACb[(size_t)(k - row0) * kSecTile + lane];
      slot = __fmaf_rn(slot, A.eta_ac, __fmul_rn(dc, A.eta_dc));
      if (A.stage == 10) A.stage_out[((int64_t)f.lam_row0 + k) * 256 + s] = dc;
    };
    if (A.dc_uniform) {
      // tiles start on multiples of 32 rows, so every 32-row block opens on
      // an anchor row
      const float d = bdc[0];
      const float* col = DS + lane;
      for (int kb = row0 + warp * kDcAnchor; kb < k_hi; kb += kIhcWarps * kDcAnchor) {
        const int ke = min(kb + kDcAnchor, k_hi);
        float ws = 0.0f, wc = 0.0f;
        int tu_prev = -1;
        // taps_used(k) stepped from row to row: lim = (k + 1) mod sg(k)
        int sg = kb < f.frdp - 1 ? f.seg : f.total;
        int lim = (kb + 1) % sg;
#pragma unroll 4
        for (int k = kb; k < ke; ++k) {
          const int tu = lim < A.n_dc ? lim : A.n_dc;
          // both window ends lie inside DS for every tu <= n_dc, so they are
          // loaded ahead of the dependent sums
          const float x_new = col[(size_t)(k - dsbase) * kSecTile];
          const float x_old = col[(size_t)(k - tu - dsbase) * kSecTile];
          if (k == kb || (tu != tu_prev && tu != tu_prev + 1)) {
            ws = wc = 0.0f;
            for (int j = 0; j < tu; ++j)
              two_sum_add(ws, wc, col[(size_t)(k - j - dsbase) * kSecTile]);
          } else {
            two_sum_add(ws, wc, x_new);
            if (tu == tu_prev) two_sum_add(ws, wc, -x_old);
          }
          tu_prev = tu;
          if (k + 1 == f.frdp - 1) {
            sg = f.total;
            lim = (k + 2) % sg;
          } else if (++lim == sg) {
            lim = 0;
          }
          // d * (ws + wc), rounded once
          const float p = __fmul_rn(d, ws);
          const float q = __fmaf_rn(d, ws, -p);
          set_pre(k, __fadd_rn(p, __fmaf_rn(d, wc, q)));
        }
      }
    } else {
      for (int kb = row0 + warp * kRB; kb < k_hi; kb += kIhcWarps * kRB) {
        const int nr = min(kRB, k_hi - kb);
        bool fast = nr == kRB;
#pragma unroll
        for (int r = 0; r < kRB; ++r)
          fast = fast && taps_used(kb + r, f, A.n_dc) == A.n_dc;
        float acc[kRB];
        const float* src = DS + (size_t)(kb - dsbase) * kSecTile + lane;
        if (fast) {
          fir_block8(src, bdc, A.n_dc, acc);
        } else {
#pragma unroll
          for (int r = 0; r < kRB; ++r)
            acc[r] = r < nr ? fir_row(src + r * kSecTile, bdc, taps_used(kb + r, f, A.n_dc))
                            : 0.0f;
        }
#pragma unroll
        for (int r = 0; r < kRB; ++r)
          if (r < nr) set_pre(kb + r, acc[r]);
      }
    }
    __syncthreads();
    for (int kb = row0 + warp * kEmitRows; kb < k_hi; kb += kIhcWarps * kEmitRows) {
      float lg[kEmitRows], l0[kEmitRows], l1[kEmitRows], l2[kEmitRows];
#pragma unroll
      for (int r = 0; r < kEmitRows; ++r) {
        // rows past the tile repeat its last row; they are not stored
        const int k = min(kb + r, k_hi - 1);
        const float pre = ACb[(size_t)(k - row0) * kSecTile + lane];
        const float y = __fmul_rn(dmg, pre);
        lg[r] = own_log10f(__fadd_rn(fmaxf(y, 0.0f), 1e-20f));
        l0[r] = sec0 ? A.spont0 : fminf(A.sat, fmaxf(__fmul_rn(a0, lg[r]), A.spont0));
        l1[r] = sec0 ? A.spont1 : fminf(A.sat, fmaxf(__fmul_rn(a1, lg[r]), A.spont1));
        l2[r] = sec0 ? A.spont2 : fminf(A.sat, fmaxf(__fmul_rn(a2, lg[r]), A.spont2));
      }
#pragma unroll
      for (int r = 0; r < kEmitRows; ++r) {
        if (kb + r < k_hi) {
          const int64_t row = f.lam_row0 + kb + r;
          A.lam[(0 * A.lam_plane_rows + row) * 256 + s] = l0[r];
          A.lam[(1 * A.lam_plane_rows + row) * 256 + s] = l1[r];
          A.lam[(2 * A.lam_plane_rows + row) * 256 + s] = l2[r];
          if (A.ihc) A.ihc[row * 256 + s] = lg[r];
          if (A.lam_host) {
            A.lam_host[(0 * A.lam_plane_rows + row) * 256 + s] = l0[r];
            A.lam_host[(1 * A.lam_plane_rows + row) * 256 + s] = l1[r];
            A.lam_host[(2 * A.lam_plane_rows + row) * 256 + s] = l2[r];
          }
        }
      }
    }
    __syncthreads();
  }
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

size_t smem_bytes(int TR, int xrows, int n_ac, int n_dc) {
  return ((size_t)xrows + TR + n_dc + TR) * kSecTile * 4 + (size_t)(n_ac + n_dc) * 4 + 32;
}

// Output rows per tile: a multiple of 32 (the DC anchor grid) whose staged
// window fits 227 KB of shared memory, at most 384.  Preferred: the largest
// such TR that is a multiple of kIhcWarps * kRB (every warp gets the same
// number of register blocks in phase 1) and >= n_dc (runs of tiles); else
// the largest that fits.  TR = 0: the filters are too long for one tile.
void pick_tile(int n_ac, int n_dc, int* TR, int* xrows) {
  *TR = *xrows = 0;
  int any = 0, ax = 0;
  for (int tr = 384; tr >= 32; tr -= 32) {
    const int xr = (tr + n_ac + n_dc - 1 + kBoxRows - 1) / kBoxRows * kBoxRows;
    if (smem_bytes(tr, xr, n_ac, n_dc) > 227 * 1024) continue;
    if (!any) {
      any = tr;
      ax = xr;
    }
    if (tr % (kIhcWarps * kRB) == 0 && tr >= n_dc) {
      *TR = tr;
      *xrows = xr;
      return;
    }
  }
  *TR = any;
  *xrows = ax;
}

// The AC taps as the kernel uses them (scaled in float) are symmetric,
// b_k == b_{n-1-k}: the FIR then runs over tap pairs (fir_block8_sym).
int ac_symmetric(const float* ac_taps, int n_ac, float scale) {
  if (n_ac < 2) return 0;
  for (int i = 0; i < n_ac / 2; ++i)
    if (ac_taps[i] * scale != ac_taps[n_ac - 1 - i] * scale) return 0;
  return 1;
}

// Tiles per CTA run of the FP32 kernel.  A run's first tile recomputes the DC filter's n_dc - 1
// look-back rows, so longer runs cost less; the longest of 32 and 16 tiles
// that still leaves at least two CTAs per SM (eight section blocks per run),
// else 8.  Runs need TR >= n_dc (the look-back is inherited in place).  The
// choice depends only on the frame table and the device, so the upload and
// the launch of one table agree.
// Tiles per run forced by cgb_ihc_set_run_length (the autotuner), 0: the rule below.
int g_forced_run = 0;

// How each scratch buffer's tables were uploaded: the tile prefix on the device
// depends on the kernel and the run length, so a launch of uploaded tables must
// use the same ones whatever the settings are by then, and what the kernels take
// from the taps is of the uploaded ones.  A launch with other lengths would read
// the tables at the wrong places: it is an error.
struct Uploaded {
  int n_frames, n_ac, n_dc;
  int n_tiles;  // runs of tiles of all frames
  int run;
  bool tensor;
  TensorTaps taps;
  int ac_sym, dc_uniform;
};
std::mutex g_uploaded_mu;
std::unordered_map<const void*, Uploaded> g_uploaded;

int sm_count() {
  int dev = 0, n_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  return n_sm;
}

// The tensor kernel's run: each CTA (one per SM) takes the time of its tiles and
// of the two before the first that the DC filter looks back on, and the CTAs
// go in waves over the SMs; the length with the least waves x tiles.
int pick_tensor_run(const cgb_ihc_frame* frames, int n_frames, int n_dc) {
  if (g_forced_run > 0) return g_forced_run;
  const int n_sm = std::max(1, sm_count());
  const long long back = (n_dc - 1 + kTensorTileRows - 1) / kTensorTileRows;
  int best = 1;
  long long best_cost = 0;
  for (int r : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64}) {
    long long runs = 0;
    for (int i = 0; i < n_frames; ++i) {
      const long long tiles = ((long long)frames[i].lam_rows + kTensorTileRows - 1) /
                              kTensorTileRows;
      runs += (tiles + r - 1) / r;
    }
    const long long ctas = runs * (256 / kTensorSections);
    const long long cost = (ctas + n_sm - 1) / n_sm * (r + back);
    if (r == 1 || cost < best_cost) {
      best = r;
      best_cost = cost;
    }
  }
  return best;
}

int pick_run(const cgb_ihc_frame* frames, int n_frames, int TR, int n_dc) {
  if (TR < n_dc) return 1;
  if (g_forced_run > 0) return g_forced_run;
  int n_sm = sm_count();
  if (n_sm < 1) n_sm = 1 << 20;  // unknown: keep the short runs
  for (int r : {32, 16}) {
    long long runs = 0;
    for (int i = 0; i < n_frames; ++i) {
      const long long tiles = ((long long)frames[i].lam_rows + TR - 1) / TR;
      runs += (tiles + r - 1) / r;
    }
    if (runs * (256 / kSecTile) >= 2LL * n_sm) return r;
  }
  return kTilesPerRun;
}

// Whether the tensor kernel is the faster one for these frames.  It takes whole tiles of
// 128 rows, rows or not, at the same time for all of its filters, and evaluates the rows
// behind a segment's end inside a tile one by one; the FP32 kernel's time goes with the
// rows and their taps, and its CTAs have half as many sections, which counts while the
// chip is not full.  Times in us of an SM for 64 sections, fitted to (FP32 / tensor, us)
//   600 frames of 100 rows, 64 taps: 614 / 650, 255 taps: 740 / 650; 2,400 of 25: 1,381 /
//   2,260; 200 of 300: 450 / 557, 1,204 / 601; 60 of 1,000: 523 / 455, 1,412 / 481; 3 of
//   100: 35 / 54; one of 30: 25 / 49; one of 60,000 in segments of 50 (255 taps): 435 / 755,
//   100: 696 / 846, 200: 1,122 / 792; 2.9 million rows, 64 taps: 19,200 / 17,100.
bool tensor_faster(const cgb_ihc_frame* frames, int n_frames, int n_ac, int n_dc, int TR,
                   int run, int tensor_run) {
  const double back = (n_dc - 1 + kTensorTileRows - 1) / kTensorTileRows;
  double all = 0.0, all_t = 0.0, one = 0.0, one_t = 0.0;  // of all CTAs, of the longest
  double ctas = 0.0, ctas_t = 0.0;
  for (int i = 0; i < n_frames; ++i) {
    const cgb_ihc_frame& f = frames[i];
    if (f.lam_rows <= 0 || f.seg <= 0) continue;
    const double rows = f.lam_rows, len = std::min(f.seg, f.lam_rows), segs = rows / len;
    const double part = std::min(len, (double)n_ac);  // rows of a segment with fewer taps
    const double row = 0.075 + (4.5e-3 * part * part / 2 + 2.75e-3 * n_ac * (len - part)) / len;
    const double runs = std::ceil(rows / ((double)run * TR));
    ctas += runs * (256 / kSecTile);
    all += 21.0 * runs + row * rows;
    one = std::max(one, 21.0 + row * std::min(rows, (double)run * TR + (runs > 1 ? n_dc : 0)));
    const double tiles = std::ceil(rows / kTensorTileRows);
    const double runs_t = std::ceil(tiles / tensor_run);
    const double cut = f.seg % kTensorTileRows ? std::min(len, kTensorTileRows / 2.0) : 0.0;
    const double tile = 27.0 + 5e-3 * (segs - 1) / tiles * cut * cut;
    ctas_t += runs_t * (256 / kTensorSections);
    all_t += 14.0 * runs_t + tile * (tiles + (runs_t - 1) * back);
    one_t = std::max(one_t, 14.0 + tile * (std::min(tiles, (double)tensor_run) +
                                           (runs_t > 1 ? back : 0)));
  }
  const double sms = std::max(1, sm_count());
  // few CTAs go in whole waves
  auto time = [&](double total, double longest, double n) {
    return n <= 4 * sms ? std::ceil(n / sms) * longest : std::max(4 * total / sms, longest);
  };
  return 1.05 * time(all_t, one_t, ctas_t) < time(all, one / 2, ctas);
}

}  // namespace
}  // namespace cgb

namespace cgb {
// bytes of the per-call tables: frames, tile prefix, taps, each 256-aligned
constexpr int64_t ihc_table_bytes(int n_frames, int n_taps) {
  return ((int64_t)n_frames * (int64_t)sizeof(cgb_ihc_frame) + 255) / 256 * 256 +
         ((int64_t)(n_frames + 1) * 4 + 255) / 256 * 256 + ((int64_t)n_taps * 4 + 255) / 256 * 256;
}
}  // namespace cgb

extern "C" int64_t cgb_ihc_lambda_scratch_bytes(int n_frames, int n_ac, int n_dc) {
  return cgb::ihc_table_bytes(n_frames, n_ac + n_dc);
}

namespace cgb {
namespace {
constexpr int kUpload = 1, kLaunch = 2;

// Validates the frame table, then uploads the per-call tables (frames, tile
// prefix, taps) to the scratch buffer (kUpload) and/or launches the kernel
// on tables already there (kLaunch).  Upload and launch are separable so a
// CUDA graph can capture the launch alone.
int ihc_lambda_impl(const float* d_v, int64_t v_rows, const cgb_ihc_frame* frames, int n_frames,
                    const float* ac_taps, int n_ac, const float* dc_taps, int n_dc,
                    const cgb_ihc_params* prm, const float* d_dmg, int n_dmg_profiles,
                    const float* d_aihc, float* d_lam, int64_t lam_plane_rows, float* d_ihc,
                    void* d_scratch, int64_t scratch_bytes, int32_t* d_status, void* stream,
                    int mode,
                    const float* ac_ext = nullptr, float* lam_host = nullptr,
                    int32_t* stage_prefix = nullptr, float* stage_taps = nullptr,
                    int stage = 0, float* d_stage = nullptr) {
  if (n_frames == 0) return CGB_OK;
  if (!frames || n_frames < 0 || !ac_taps || !dc_taps || !prm || !d_scratch ||
      ((mode & kLaunch) && (!d_v || !d_dmg || !d_aihc || !d_lam || !d_status)))
    return fail(CGB_ERR_ARG, "cgb_ihc_lambda_dev: null pointer argument");
  if (n_ac < 1 || n_dc < 1 || n_ac > 1024 || n_dc > 1024)
    return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_dev: filter lengths must be in [1, 1024]");
  if (scratch_bytes < cgb_ihc_lambda_scratch_bytes(n_frames, n_ac, n_dc))
    return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_dev: scratch buffer too small");
  if ((mode & kLaunch) && (reinterpret_cast<uintptr_t>(d_v) & 15))
    return fail(CGB_ERR_ARG, "cgb_ihc_lambda_dev: d_v must be 16-byte aligned");
  if (lam_host) {
    const int rc = check_host_mirror(lam_host, "cgb_ihc_lambda_dev: h_lam");
    if (rc) return rc;
  }
  if (stage != 0 && (stage < 9 || stage > 12 || ((mode & kLaunch) && !d_stage)))
    return fail(CGB_ERR_ARG, "cgb_ihc_lambda_stage_dev: stage must be 9-12 with an output buffer");
  if (v_rows > INT32_MAX)
    return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_dev: more than 2^31-1 velocity rows");
  // host staging of the tile prefix and the taps: a vector, or the caller's
  // fixed arrays (stage_prefix: n_frames + 1 entries, stage_taps: n_ac + n_dc)
  std::vector<int32_t> prefix_v;
  int32_t* prefix = stage_prefix;
  if (!prefix) {
    prefix_v.assign(n_frames + 1, 0);
    prefix = prefix_v.data();
  }
  prefix[0] = 0;
  int TR = 0, xrows = 0;
  pick_tile(n_ac, n_dc, &TR, &xrows);
  if (TR < 32) return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_dev: filters too long for one tile");
  Uploaded up{};
  bool known = false;
  if (!(mode & kUpload)) {
    std::lock_guard<std::mutex> lock(g_uploaded_mu);
    const auto it = g_uploaded.find(d_scratch);
    known = it != g_uploaded.end();
    if (known) up = it->second;
  }
  if (!known) {
    up = {n_frames, n_ac, n_dc, 0, pick_run(frames, n_frames, TR, n_dc), false, {},
          ac_symmetric(ac_taps, n_ac, prm->scale), 1};
    for (int i = 1; i < n_dc; ++i) up.dc_uniform &= dc_taps[i] == dc_taps[0];
    // The AC filter goes to the tensor cores where the kernel is built for it (a uniform DC
    // filter, no debug stage, no AC given, lengths that fit) and the faster one.
    if (!ac_ext && stage == 0 && up.dc_uniform && ihc_tensor_fits(n_ac, n_dc) &&
        ihc_tensor_taps(ac_taps, n_ac, prm->scale, &up.taps)) {
      const int run = pick_tensor_run(frames, n_frames, n_dc);
      up.tensor = tensor_faster(frames, n_frames, n_ac, n_dc, TR, up.run, run);
      if (up.tensor) up.run = run;
    }
  }
  if (up.n_ac != n_ac || up.n_dc != n_dc)
    return fail(CGB_ERR_ARG, "cgb_ihc_lambda_launch_dev: not the filters that were uploaded");
  if (up.n_frames != n_frames)
    return fail(CGB_ERR_ARG, "cgb_ihc_lambda_launch_dev: not the frames that were uploaded");
  if (up.tensor) TR = kTensorTileRows;
  for (int i = 0; i < n_frames; ++i) {
    const cgb_ihc_frame& fr = frames[i];
    const bool ok = fr.v_row0 >= 0 && fr.lam_rows >= 0 && fr.lam_rows <= fr.rows &&
                    fr.v_row0 + fr.rows <= v_rows && fr.lam_row0 >= 0 &&
                    fr.lam_row0 + fr.lam_rows <= lam_plane_rows && fr.seg > 0 && fr.frdp > 0 &&
                    fr.total > 0 && fr.ihc_profile >= 0 && fr.ihc_profile < n_dmg_profiles;
    if (!ok)
      return fail(CGB_ERR_RANGE,
                  "cgb_ihc_lambda_dev: frame " + std::to_string(i) + " out of range");
    const int tiles = (fr.lam_rows + TR - 1) / TR;
    prefix[i + 1] = prefix[i] + (tiles + up.run - 1) / up.run;
  }
  const int n_tiles = prefix[n_frames];
  if (known && n_tiles != up.n_tiles)
    return fail(CGB_ERR_ARG, "cgb_ihc_lambda_launch_dev: not the frames that were uploaded");
  up.n_tiles = n_tiles;
  if (mode & kUpload) {
    std::lock_guard<std::mutex> lock(g_uploaded_mu);
    g_uploaded[d_scratch] = up;
  }
  if (n_tiles == 0) return CGB_OK;

  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  unsigned char* sc = static_cast<unsigned char*>(d_scratch);
  const size_t fbytes = ((size_t)n_frames * sizeof(cgb_ihc_frame) + 255) / 256 * 256;
  const size_t pbytes = ((size_t)(n_frames + 1) * 4 + 255) / 256 * 256;
  if (mode & kUpload) {
    std::vector<float> taps_v;
    float* taps = stage_taps;
    if (!taps) {
      taps_v.resize(n_ac + n_dc);
      taps = taps_v.data();
    }
    for (int i = 0; i < n_ac; ++i) taps[i] = ac_taps[i] * prm->scale;
    for (int i = 0; i < n_dc; ++i) taps[n_ac + i] = dc_taps[i];
    CGB_TRY_CUDA(cudaMemcpyAsync(sc, frames, (size_t)n_frames * sizeof(cgb_ihc_frame),
                                 cudaMemcpyHostToDevice, st),
                 "upload frames");
    CGB_TRY_CUDA(cudaMemcpyAsync(sc + fbytes, prefix, (size_t)(n_frames + 1) * 4,
                                 cudaMemcpyHostToDevice, st),
                 "upload tile prefix");
    CGB_TRY_CUDA(cudaMemcpyAsync(sc + fbytes + pbytes, taps, (size_t)(n_ac + n_dc) * 4,
                                 cudaMemcpyHostToDevice, st),
                 "upload taps");
  }
  if (!(mode & kLaunch)) return CGB_OK;

  IHCArgs A{};
  A.frames = reinterpret_cast<const cgb_ihc_frame*>(sc);
  A.tile_prefix = reinterpret_cast<const int32_t*>(sc + fbytes);
  A.n_frames = n_frames;
  A.taps = reinterpret_cast<const float*>(sc + fbytes + pbytes);
  A.n_ac = n_ac;
  A.n_dc = n_dc;
  A.scale = prm->scale;
  A.eta_ac = prm->eta_ac;
  A.eta_dc = prm->eta_dc;
  A.sat = prm->lambda_sat;
  A.spont0 = prm->spont[0];
  A.spont1 = prm->spont[1];
  A.spont2 = prm->spont[2];
  A.dmg = d_dmg;
  A.aihc = d_aihc;
  A.lam = d_lam;
  A.lam_host = lam_host;
  A.lam_plane_rows = lam_plane_rows;
  A.ihc = d_ihc;
  A.TR = TR;
  A.xrows = xrows;
  A.status = d_status;
  A.ac_ext = ac_ext;
  A.skip_first_copy = g_fault_skip_copy;
  A.stage = stage == 12 ? 11 : stage;  // the reference's 12 ("Shigh") is dS too
  A.stage_out = d_stage;
  A.run = up.run;
  A.dc_uniform = up.dc_uniform;
  A.ac_sym = up.ac_sym;
  if (up.tensor) return ihc_tensor_launch(A, d_v, n_tiles, up.taps, st);

  CUtensorMap map;
  auto encode = get_encode();
  if (!encode) return fail(CGB_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[2] = {256, (cuuint64_t)v_rows};
  cuuint64_t strides[1] = {256 * 4};
  cuuint32_t box[2] = {(cuuint32_t)kSecTile, (cuuint32_t)kBoxRows};
  cuuint32_t estr[2] = {1, 1};
  CUresult cr = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(d_v), dims,
                       strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS)
    return fail(CGB_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)cr) + ")");

  const size_t smem = smem_bytes(TR, xrows, n_ac, n_dc);
  CGB_TRY_CUDA(cudaFuncSetAttribute(ihc_lambda_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "cudaFuncSetAttribute(ihc smem)");
  dim3 grid((unsigned)n_tiles, 256 / kSecTile);
  ihc_lambda_kernel<<<grid, kIhcWarps * 32, smem, st>>>(map, A);
  CGB_TRY_CUDA(cudaGetLastError(), "ihc_lambda_kernel launch");
  note_launch();
  return CGB_OK;
}

}  // namespace
}  // namespace cgb

extern "C" int cgb_ihc_set_run_length(int tiles) {
  if (tiles < 0 || tiles > 64)
    return cgb::fail(CGB_ERR_ARG, "cgb_ihc_set_run_length: tiles must be 0 (automatic) or 1-64");
  cgb::g_forced_run = tiles;
  return CGB_OK;
}

extern "C" int cgb_ihc_set_fault_injection(int skip_first_copy) {
  cgb::g_fault_skip_copy = skip_first_copy ? 1 : 0;
  return CGB_OK;
}

extern "C" int cgb_ihc_lambda_dev(const float* d_v, int64_t v_rows, const cgb_ihc_frame* frames,
                                  int n_frames, const float* ac_taps, int n_ac,
                                  const float* dc_taps, int n_dc, const cgb_ihc_params* prm,
                                  const float* d_dmg, int n_dmg_profiles, const float* d_aihc,
                                  float* d_lam, int64_t lam_plane_rows, float* d_ihc,
                                  void* d_scratch, int64_t scratch_bytes, int32_t* d_status,
                                  void* stream) {
  return cgb::ihc_lambda_impl(d_v, v_rows, frames, n_frames, ac_taps, n_ac, dc_taps, n_dc, prm,
                              d_dmg, n_dmg_profiles, d_aihc, d_lam, lam_plane_rows, d_ihc,
                              d_scratch, scratch_bytes, d_status, stream,
                              cgb::kUpload | cgb::kLaunch);
}

extern "C" int cgb_ihc_lambda_stage_dev(const float* d_v, int64_t v_rows,
                                        const cgb_ihc_frame* frames, int n_frames,
                                        const float* ac_taps, int n_ac, const float* dc_taps,
                                        int n_dc, const cgb_ihc_params* prm, const float* d_dmg,
                                        int n_dmg_profiles, const float* d_aihc, float* d_lam,
                                        int64_t lam_plane_rows, float* d_ihc, int stage,
                                        float* d_stage, void* d_scratch, int64_t scratch_bytes,
                                        int32_t* d_status, void* stream) {
  if (stage < 9 || stage > 12 || !d_stage)
    return cgb::fail(CGB_ERR_ARG,
                     "cgb_ihc_lambda_stage_dev: stage must be 9-12 with an output buffer");
  return cgb::ihc_lambda_impl(d_v, v_rows, frames, n_frames, ac_taps, n_ac, dc_taps, n_dc, prm,
                              d_dmg, n_dmg_profiles, d_aihc, d_lam, lam_plane_rows, d_ihc,
                              d_scratch, scratch_bytes, d_status, stream,
                              cgb::kUpload | cgb::kLaunch, nullptr, nullptr, nullptr, nullptr,
                              stage, d_stage);
}

extern "C" int cgb_ihc_lambda_upload_dev(const cgb_ihc_frame* frames, int n_frames,
                                         const float* ac_taps, int n_ac, const float* dc_taps,
                                         int n_dc, const cgb_ihc_params* prm, int64_t v_rows,
                                         int64_t lam_plane_rows, int n_dmg_profiles,
                                         void* d_scratch, int64_t scratch_bytes, void* stream) {
  return cgb::ihc_lambda_impl(nullptr, v_rows, frames, n_frames, ac_taps, n_ac, dc_taps, n_dc,
                              prm, nullptr, n_dmg_profiles, nullptr, nullptr, lam_plane_rows,
                              nullptr, d_scratch, scratch_bytes, nullptr, stream, cgb::kUpload);
}

extern "C" int cgb_ihc_lambda_launch_dev(const float* d_v, int64_t v_rows,
                                         const cgb_ihc_frame* frames, int n_frames,
                                         const float* ac_taps, int n_ac, const float* dc_taps,
                                         int n_dc, const cgb_ihc_params* prm,
                                         const float* d_dmg, int n_dmg_profiles,
                                         const float* d_aihc, float* d_lam,
                                         int64_t lam_plane_rows, float* d_ihc, void* d_scratch,
                                         int64_t scratch_bytes, int32_t* d_status, void* stream) {
  return cgb::ihc_lambda_impl(d_v, v_rows, frames, n_frames, ac_taps, n_ac, dc_taps, n_dc, prm,
                              d_dmg, n_dmg_profiles, d_aihc, d_lam, lam_plane_rows, d_ihc,
                              d_scratch, scratch_bytes, d_status, stream, cgb::kLaunch);
}

extern "C" int cgb_ihc_lambda_launch_mirror_dev(
    const float* d_v, int64_t v_rows, const cgb_ihc_frame* frames, int n_frames,
    const float* ac_taps, int n_ac, const float* dc_taps, int n_dc, const cgb_ihc_params* prm,
    const float* d_dmg, int n_dmg_profiles, const float* d_aihc, float* d_lam,
    int64_t lam_plane_rows, float* d_ihc, void* d_scratch, int64_t scratch_bytes,
    int32_t* d_status, float* h_lam, int64_t h_lam_bytes, void* stream) {
  if (!h_lam) return cgb::fail(CGB_ERR_ARG, "cgb_ihc_lambda_launch_mirror_dev: null h_lam");
  if (h_lam_bytes < 3 * lam_plane_rows * 256 * (int64_t)sizeof(float))
    return cgb::fail(CGB_ERR_RANGE, "cgb_ihc_lambda_launch_mirror_dev: h_lam is shorter than "
                                    "3 x lam_plane_rows x 256 floats");
  return cgb::ihc_lambda_impl(d_v, v_rows, frames, n_frames, ac_taps, n_ac, dc_taps, n_dc, prm,
                              d_dmg, n_dmg_profiles, d_aihc, d_lam, lam_plane_rows, d_ihc,
                              d_scratch, scratch_bytes, d_status, stream, cgb::kLaunch, nullptr,
                              h_lam);
}

// ---------------------------------------------------------------------------
// No-allocation variant of cgb_ihc_lambda_dev.
//
// The per-call tables (frames, tile prefix, filter taps) go to a file-scope
// __device__ array instead of caller scratch, for callers that cannot
// allocate device memory: a host that hands the library only the buffers it
// already owns, or a real-time audio thread that must not enter the device
// allocator (nor the host heap: the host-side staging of the prefix and taps
// is a pair of static arrays too).  The array is 192 KiB, holds at most
// kNoAllocMaxFrames frames and kNoAllocMaxTaps taps, and stays resident on
// every GPU that loads this library until the process exits.  All calls
// share it and the static staging, so calls must come from one host thread
// at a time and calls whose GPU work overlaps (different streams, or a
// second call enqueued before the first one ran) race on its contents;
// serialise them on one stream.  Each call rewrites every table byte it
// reads, so nothing needs clearing.  The tables are the same layout as the
// caller-scratch path's (frames, then the prefix, then the taps, each
// 256-byte aligned), sized for the maximum.
// ---------------------------------------------------------------------------
namespace cgb {
namespace {

constexpr int kNoAllocMaxFrames = 4096;
constexpr int kNoAllocMaxTaps = 2048;  // n_ac + n_dc
constexpr size_t kNoAllocBytes = 192 * 1024;
static_assert((size_t)ihc_table_bytes(kNoAllocMaxFrames, kNoAllocMaxTaps) <= kNoAllocBytes,
              "no-allocation scratch too small");

__device__ __align__(256) unsigned char g_ihc_noalloc_scratch[kNoAllocBytes];

// host staging of the tile prefix and the taps (no heap use per call)
int32_t g_noalloc_prefix[kNoAllocMaxFrames + 1];
float g_noalloc_taps[kNoAllocMaxTaps];

constexpr int kMaxDevices = 64;
std::atomic<void*> g_noalloc_ptr[kMaxDevices] = {};

// Device address of the array on the current device, looked up once per
// device (the host-side symbol is only a stand-in, not a device address).
// Concurrent first calls may both look it up; they store the same address.
// The cache is not cleared by cudaDeviceReset: after a reset, a process that
// calls this entry point again must be a new process.
int noalloc_scratch(void** out) {
  int dev = 0;
  CGB_TRY_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices)
    return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_noalloc_dev: device index beyond 63");
  void* p = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (!p) {
    CGB_TRY_CUDA(cudaGetSymbolAddress(&p, g_ihc_noalloc_scratch), "cudaGetSymbolAddress");
    g_noalloc_ptr[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return CGB_OK;
}

}  // namespace
}  // namespace cgb

extern "C" int cgb_ihc_lambda_noalloc_dev(const float* d_v, int64_t v_rows,
                                          const cgb_ihc_frame* frames, int n_frames,
                                          const float* ac_taps, int n_ac, const float* dc_taps,
                                          int n_dc, const cgb_ihc_params* prm,
                                          const float* d_dmg, int n_dmg_profiles,
                                          const float* d_aihc, float* d_lam,
                                          int64_t lam_plane_rows, float* d_ihc,
                                          int32_t* d_status, void* stream) {
  using namespace cgb;
  if (n_frames == 0) return CGB_OK;
  if (n_frames > kNoAllocMaxFrames)
    return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_noalloc_dev: more than 4096 frames (the fixed "
                               "scratch holds at most 4096)");
  if (n_ac < 1 || n_dc < 1 || n_ac > 1024 || n_dc > 1024 || n_ac + n_dc > kNoAllocMaxTaps)
    return fail(CGB_ERR_RANGE,
                "cgb_ihc_lambda_noalloc_dev: filter lengths must be in [1, 1024]");
  void* scratch = nullptr;
  if (int st = noalloc_scratch(&scratch)) return st;
  return ihc_lambda_impl(d_v, v_rows, frames, n_frames, ac_taps, n_ac, dc_taps, n_dc, prm,
                         d_dmg, n_dmg_profiles, d_aihc, d_lam, lam_plane_rows, d_ihc, scratch,
                         (int64_t)kNoAllocBytes, d_status, stream, kUpload | kLaunch, nullptr,
                         nullptr, g_noalloc_prefix, g_noalloc_taps);
}

// ---------------------------------------------------------------------------
// AC by IIR (the reference's is_ac_iir_filter path, DeviceCudaIIRFilter,
// src/cochlea.cu:2745-2775):
//   Y[k] = sum_{i<ob} b_i X[k-i] - sum_{1<=j<ob} a_j Y[k-j]
// with ob the FIR look-back bound.  The reference keeps Y in float (lambdaFloat)
// and adds each double-tap term in double before rounding back to float; the
// kernel performs those FP64 operations in the same order (products and sums
// rounded separately).  The recursion is sequential in time, so a CTA walks one
// segment of a frame -- rows between two points where the look-back rule gives
// zero taps, which start the recursion afresh -- for 32 sections.  A row's b
// terms come first and need no earlier output: three warps form them for the
// next rows while the fourth runs the a terms, its last outputs in registers.
//
// What bounds it: the chain of a row's a terms, each a widening, an FP64 addition
// and a rounding that wait for one another (192 cycles).  With a CTA of 256
// threads per segment it was the SM's FP64 unit under eight warps (413 cycles a
// term), and the outputs were read back from memory.  Measured (GB300), the whole
// stage from and to host arrays: four segments of 2,500 rows, order 2, 6.4 -> 2.7
// ms; order 4, 10.5 -> 2.3; one of 5,000, order 2, 9.5 -> 2.1.
// ---------------------------------------------------------------------------
namespace cgb {
namespace {

struct IIRSeg {
  int64_t v_row0;  // the frame's first velocity row
  int32_t k0, k1;  // frame rows [k0, k1)
  int32_t frame;
  int32_t pad;
};

constexpr int kIirWarps = 4;   // three for the b terms, one for the a terms
constexpr int kIirChunk = 24;  // rows of b terms formed ahead

// N: the filter's length where its N - 1 last outputs fit in registers, else 0
// (they are read back).
template <int N>
__global__ void __launch_bounds__(kIirWarps * 32)
    iir_ac_kernel(const float* __restrict__ v, float* __restrict__ ac,
                  const IIRSeg* __restrict__ segs, const cgb_ihc_frame* __restrict__ frames,
                  const double* __restrict__ b, const double* __restrict__ a, int n) {
  __shared__ float input[2][kIirChunk][32];
  const IIRSeg sg = segs[blockIdx.x];
  const cgb_ihc_frame f = frames[sg.frame];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t at = sg.v_row0 * 256 + 32 * blockIdx.y + lane;
  const float* x = v + at;
  float* y = ac + at;
  auto b_terms = [&](int chunk) {
    const int k_first = sg.k0 + chunk * kIirChunk;
    for (int q = warp - 1; q < kIirChunk && k_first + q < sg.k1; q += kIirWarps - 1) {
      const int k = k_first + q, ob = taps_used(k, f, n);
      float yk = 0.0f;
      for (int i = 0; i < ob; ++i)
        yk = __double2float_rn(
            __dadd_rn((double)yk, __dmul_rn(b[i], (double)x[(int64_t)(k - i) * 256])));
      input[chunk & 1][q][lane] = yk;
    }
  };
  double ra[N > 1 ? N : 1], past[N > 1 ? N : 1];  // past[j]: output k - j
#pragma unroll
  for (int j = 1; j < N; ++j) {
    ra[j] = a[j];
    past[j] = 0.0;
  }
  // the look-back rule stepped from row to row: lim = (k + 1) mod rule(k)
  int rule = sg.k0 < f.frdp - 1 ? f.seg : f.total;
  int lim = (sg.k0 + 1) % rule;
  const int chunks = (sg.k1 - sg.k0 + kIirChunk - 1) / kIirChunk;
  if (warp > 0) b_terms(0);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    __syncthreads();
    if (warp > 0) {
      if (chunk + 1 < chunks) b_terms(chunk + 1);
      continue;
    }
    const int k_first = sg.k0 + chunk * kIirChunk;
    const int rows = min(kIirChunk, sg.k1 - k_first);
    for (int q = 0; q < rows; ++q) {
      const int k = k_first + q, ob = lim < n ? lim : n;
      float yk = input[chunk & 1][q][lane];
      if (N > 0) {
#pragma unroll
        for (int j = 1; j < N; ++j)
          if (j < ob) yk = __double2float_rn(__dsub_rn((double)yk, __dmul_rn(ra[j], past[j])));
#pragma unroll
        for (int j = N - 1; j > 1; --j) past[j] = past[j - 1];
        if (N > 1) past[1] = (double)yk;
      } else {
        for (int j = 1; j < ob; ++j)
          yk = __double2float_rn(
              __dsub_rn((double)yk, __dmul_rn(a[j], (double)y[(int64_t)(k - j) * 256])));
      }
      y[(int64_t)k * 256] = yk;
      if (k + 1 == f.frdp - 1) {
        rule = f.total;
        lim = (k + 2) % rule;
      } else if (++lim == rule) {
        lim = 0;
      }
    }
  }
}

template <int N>
void iir_launch(const float* v, float* ac, const IIRSeg* segs, int n_segs,
                const cgb_ihc_frame* frames, const double* b, const double* a, int n,
                cudaStream_t st) {
  iir_ac_kernel<N><<<dim3((unsigned)n_segs, 8), kIirWarps * 32, 0, st>>>(v, ac, segs, frames, b,
                                                                         a, n);
}

constexpr int kMaxIIR = 64;

// Segments of every frame's lambda rows that the recursion can run
// independently: candidate starts are rows whose look-back bound is zero;
// a candidate is dropped when a later row's recursion reaches back across it
// (where the rule switches to the frame total, the bound can jump up).
std::vector<IIRSeg> iir_segments(const cgb_ihc_frame* frames, int n_frames, int n) {
  std::vector<IIRSeg> out;
  std::vector<int> starts;
  for (int fi = 0; fi < n_frames; ++fi) {
    const cgb_ihc_frame& f = frames[fi];
    starts.assign(1, 0);
    for (int k = 0; k < f.lam_rows; ++k) {
      const int sg = k < f.frdp - 1 ? f.seg : f.total;
      const int lim = (k + 1) % sg;
      const int ob = lim < n ? lim : n;
      if (ob == 0) {
        if (k > starts.back()) starts.push_back(k);
      } else if (ob >= 2) {
        const int lo = k - ob + 1;  // oldest output row this row reads
        while (starts.size() > 1 && starts.back() > lo) starts.pop_back();
      }
    }
    for (size_t i = 0; i < starts.size(); ++i) {
      const int k1 = i + 1 < starts.size() ? starts[i + 1] : f.lam_rows;
      if (k1 > starts[i]) out.push_back({f.v_row0, starts[i], k1, fi, 0});
    }
  }
  return out;
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace
}  // namespace cgb

extern "C" int64_t cgb_ihc_lambda_iir_scratch_bytes(const cgb_ihc_frame* frames, int n_frames,
                                                    int n_iir, int n_dc) {
  using namespace cgb;
  if (!frames || n_frames < 0 || n_iir < 1 || n_iir > kMaxIIR) return -1;
  const size_t segs = iir_segments(frames, n_frames, n_iir).size();
  return cgb_ihc_lambda_scratch_bytes(n_frames, 1, n_dc) +
         (int64_t)(align256(segs * sizeof(IIRSeg)) + align256((size_t)2 * n_iir * 8));
}

namespace cgb {
namespace {

int ihc_lambda_iir_impl(const float* d_v, int64_t v_rows, const cgb_ihc_frame* frames,
                        int n_frames, const float* b_taps, const float* a_taps, int n_iir,
                        const float* dc_taps, int n_dc, const cgb_ihc_params* prm,
                        const float* d_dmg, int n_dmg_profiles, const float* d_aihc,
                        float* d_lam, int64_t lam_plane_rows, float* d_ihc, float* d_ac,
                        void* d_scratch, int64_t scratch_bytes, int32_t* d_status, void* stream,
                        int stage, float* d_stage) {
  if (n_frames == 0) return CGB_OK;
  if (!frames || n_frames < 0 || !b_taps || !a_taps || !d_ac || !d_v || !prm || !d_scratch)
    return fail(CGB_ERR_ARG, "cgb_ihc_lambda_iir_dev: null pointer argument");
  if (n_iir < 1 || n_iir > kMaxIIR)
    return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_iir_dev: IIR length must be in [1, 64]");
  const int64_t need = cgb_ihc_lambda_iir_scratch_bytes(frames, n_frames, n_iir, n_dc);
  if (scratch_bytes < need)
    return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_iir_dev: scratch buffer too small");
  for (int i = 0; i < n_frames; ++i) {
    const cgb_ihc_frame& fr = frames[i];
    if (fr.v_row0 < 0 || fr.lam_rows < 0 || fr.lam_rows > fr.rows || fr.v_row0 + fr.rows > v_rows ||
        fr.seg <= 0 || fr.frdp <= 0 || fr.total <= 0)
      return fail(CGB_ERR_RANGE, "cgb_ihc_lambda_iir_dev: frame outside the velocity rows");
  }
  const std::vector<IIRSeg> segs = iir_segments(frames, n_frames, n_iir);
  const int64_t base_bytes = cgb_ihc_lambda_scratch_bytes(n_frames, 1, n_dc);
  unsigned char* sc = static_cast<unsigned char*>(d_scratch) + base_bytes;
  const size_t seg_bytes = align256(segs.size() * sizeof(IIRSeg));
  std::vector<double> taps(2 * (size_t)n_iir);
  for (int i = 0; i < n_iir; ++i) {
    taps[i] = (double)b_taps[i] * (double)prm->scale;
    taps[n_iir + i] = (double)a_taps[i];
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // the fused kernel's tables first (its frame table is the IIR kernel's too)
  const float one = 1.0f;
  int rc = ihc_lambda_impl(d_v, v_rows, frames, n_frames, &one, 1, dc_taps, n_dc, prm, d_dmg,
                           n_dmg_profiles, d_aihc, d_lam, lam_plane_rows, d_ihc, d_scratch,
                           base_bytes, d_status, stream, kUpload);
  if (rc) return rc;
  if (!segs.empty()) {
    CGB_TRY_CUDA(cudaMemcpyAsync(sc, segs.data(), segs.size() * sizeof(IIRSeg),
                                 cudaMemcpyHostToDevice, st),
                 "upload IIR segments");
    CGB_TRY_CUDA(cudaMemcpyAsync(sc + seg_bytes, taps.data(), taps.size() * 8,
                                 cudaMemcpyHostToDevice, st),
                 "upload IIR taps");
    const double* d_b = reinterpret_cast<const double*>(sc + seg_bytes);
    // orders up to 8 keep their outputs in registers
    using Launch = decltype(&iir_launch<0>);
    static const Launch kByLength[] = {iir_launch<0>, iir_launch<1>, iir_launch<2>, iir_launch<3>,
                                      iir_launch<4>, iir_launch<5>, iir_launch<6>, iir_launch<7>,
                                      iir_launch<8>, iir_launch<9>};
    kByLength[n_iir <= 9 ? n_iir : 0](d_v, d_ac, reinterpret_cast<const IIRSeg*>(sc),
                                     (int)segs.size(),
                                     reinterpret_cast<const cgb_ihc_frame*>(d_scratch), d_b,
                                     d_b + n_iir, n_iir, st);
    CGB_TRY_CUDA(cudaGetLastError(), "iir_ac_kernel launch");
    note_launch();
  }
  return ihc_lambda_impl(d_v, v_rows, frames, n_frames, &one, 1, dc_taps, n_dc, prm, d_dmg,
                         n_dmg_profiles, d_aihc, d_lam, lam_plane_rows, d_ihc, d_scratch,
                         base_bytes, d_status, stream, kLaunch, d_ac, nullptr, nullptr, nullptr,
                         stage, d_stage);
}

}  // namespace
}  // namespace cgb

extern "C" int cgb_ihc_lambda_iir_dev(const float* d_v, int64_t v_rows,
                                      const cgb_ihc_frame* frames, int n_frames,
                                      const float* b_taps, const float* a_taps, int n_iir,
                                      const float* dc_taps, int n_dc, const cgb_ihc_params* prm,
                                      const float* d_dmg, int n_dmg_profiles, const float* d_aihc,
                                      float* d_lam, int64_t lam_plane_rows, float* d_ihc,
                                      float* d_ac, void* d_scratch, int64_t scratch_bytes,
                                      int32_t* d_status, void* stream) {
  return cgb::ihc_lambda_iir_impl(d_v, v_rows, frames, n_frames, b_taps, a_taps, n_iir, dc_taps,
                                  n_dc, prm, d_dmg, n_dmg_profiles, d_aihc, d_lam,
                                  lam_plane_rows, d_ihc, d_ac, d_scratch, scratch_bytes,
                                  d_status, stream, 0, nullptr);
}

extern "C" int cgb_ihc_lambda_iir_stage_dev(const float* d_v, int64_t v_rows,
                                            const cgb_ihc_frame* frames, int n_frames,
                                            const float* b_taps, const float* a_taps, int n_iir,
                                            const float* dc_taps, int n_dc,
                                            const cgb_ihc_params* prm, const float* d_dmg,
                                            int n_dmg_profiles, const float* d_aihc,
                                            float* d_lam, int64_t lam_plane_rows, float* d_ihc,
                                            float* d_ac, int stage, float* d_stage,
                                            void* d_scratch, int64_t scratch_bytes,
                                            int32_t* d_status, void* stream) {
  if (stage < 9 || stage > 12 || !d_stage)
    return cgb::fail(CGB_ERR_ARG,
                     "cgb_ihc_lambda_iir_stage_dev: stage must be 9-12 with an output buffer");
  return cgb::ihc_lambda_iir_impl(d_v, v_rows, frames, n_frames, b_taps, a_taps, n_iir, dc_taps,
                                  n_dc, prm, d_dmg, n_dmg_profiles, d_aihc, d_lam,
                                  lam_plane_rows, d_ihc, d_ac, d_scratch, scratch_bytes,
                                  d_status, stream, stage, d_stage);
}
