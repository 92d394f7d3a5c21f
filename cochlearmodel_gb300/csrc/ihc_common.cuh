// What the IHC / lambda kernels (ihc_lambda.cu on the FP32 pipe, ihc_tensor.cu
// with the AC filter on the tensor cores) share.
#pragma once

#include <cuda_runtime.h>

#include "cgb_device.cuh"
#include "cochlea_gb300.h"

namespace cgb {

constexpr int kSecTile = 32;   // sections per CTA (one per lane)
constexpr int kIhcWarps = 16;
// bound on one staging wait, in nanoseconds of the GPU's global timer
constexpr unsigned long long kWaitNs = 1000000000ull;

struct IHCArgs {
  const cgb_ihc_frame* frames;
  const int32_t* tile_prefix;  // [n_frames + 1] runs of tiles before each frame
  int n_frames;
  const float* taps;           // [n_ac] AC taps (x scale) then [n_dc] DC taps
  int n_ac, n_dc;
  float scale, eta_ac, eta_dc, sat;
  float spont0, spont1, spont2;
  const float* dmg;            // [P][256] 10^ihc
  const float* aihc;           // [3][256]
  float* lam;                  // [3][lam_plane_rows][256]
  float* lam_host;             // host mirror of lam (pinned, mapped), or null
  int64_t lam_plane_rows;
  float* ihc;                  // [lam rows][256] or null
  int TR, xrows;               // output rows per tile, staged rows (multiple of 64)
  int32_t* status;
  int dc_uniform;              // all DC taps equal: running window sum
  int ac_sym;                  // AC taps symmetric: FIR over tap pairs
  int run;                     // tiles per CTA (consecutive, one frame)
  const float* ac_ext;         // AC by velocity row (the IIR path), or null: the FIR
  int skip_first_copy;         // test-only: arm the first staging wait but issue no copy
  // RunIHCKernel's debug stage: 9 AC, 10 DC, 11 dS (0 none), stored by lambda
  // row into stage_out [lam rows][256]
  int stage;
  float* stage_out;
};

__device__ __forceinline__ int taps_used(int k, const cgb_ihc_frame& f, int taps) {
  const int sg = k < f.frdp - 1 ? f.seg : f.total;
  const int lim = (k + 1) % sg;
  return lim < taps ? lim : taps;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Compensated tap accumulation (Ogita-Rump-Oishi Dot2): the product error
// comes from one FMA, the sum error from TwoSum, and both are carried in c.
// The result equals the dot product evaluated in about twice the working
// precision and rounded once -- what the reference's double accumulators
// give after their float store -- at FP32 instruction rates.
struct Dot2 {
  float s, c;
  __device__ __forceinline__ void init() { s = c = 0.0f; }
  __device__ __forceinline__ void add(float b, float x) {
    const float p = __fmul_rn(b, x);
    const float q = __fmaf_rn(b, x, -p);
    const float t = __fadd_rn(s, p);
    const float z = __fsub_rn(t, s);
    const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(p, z));
    s = t;
    c = __fadd_rn(c, __fadd_rn(e, q));
  }
  // b (x1 + x2) for a symmetric tap pair: the pair sum by TwoSum, Dot2 on
  // its rounded value, b times its rounding error into c by one fma
  __device__ __forceinline__ void add_pair(float b, float x1, float x2) {
    const float sg = __fadd_rn(x1, x2);
    const float zz = __fsub_rn(sg, x1);
    const float ep = __fadd_rn(__fsub_rn(x1, __fsub_rn(sg, zz)), __fsub_rn(x2, zz));
    add(b, sg);
    c = __fmaf_rn(b, ep, c);
  }
  __device__ __forceinline__ float result() const { return __fadd_rn(s, c); }
};

// Dot2 on two independent sums at once (two-wide FP32); each element
// performs exactly the scalar Dot2 sequence.
struct Dot2x2 {
  float2 s, c;
  __device__ __forceinline__ void init() { s = c = f2b(0.0f); }
  __device__ __forceinline__ void add(float2 b, float2 x) {
    const float2 p = mul2(b, x);
    const float2 q = fma2(b, x, neg2(p));
    const float2 t = add2(s, p);
    const float2 z = sub2(t, s);
    const float2 e = add2(sub2(s, sub2(t, z)), sub2(p, z));
    s = t;
    c = add2(c, add2(e, q));
  }
  __device__ __forceinline__ void add_pair(float2 b, float2 x1, float2 x2) {
    const float2 sg = add2(x1, x2);
    const float2 zz = sub2(sg, x1);
    const float2 ep = add2(sub2(x1, sub2(sg, zz)), sub2(x2, zz));
    add(b, sg);
    c = fma2(b, ep, c);
  }
  __device__ __forceinline__ float2 result() const { return add2(s, c); }
};

// s + c += x exactly (Knuth's TwoSum; the rounding error goes to c).
__device__ __forceinline__ void two_sum_add(float& s, float& c, float x) {
  const float t = __fadd_rn(s, x);
  const float z = __fsub_rn(t, s);
  const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z));
  s = t;
  c = __fadd_rn(c, e);
}

constexpr int kDcAnchor = 32;  // DC window re-summed at frame rows k % 32 == 0
constexpr int kEmitRows = 4;   // rows per warp in one IHC / lambda batch

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar, int arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(arrivals));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}
// Whether completion `phase` (from 0) of mbar has come; the instruction waits a short
// time for it.
__device__ __forceinline__ bool mbar_done(uint64_t* mbar, int phase) {
  uint32_t done;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(done)
      : "r"(smem_u32(mbar)), "r"((uint32_t)(phase & 1))
      : "memory");
  return done != 0;
}

// Wait on phase `parity` of mbar by every thread, for at most kWaitNs of the
// global timer (each try_wait returns within a short system-defined time),
// then a block-wide vote so that all threads take the same branch.
__device__ __forceinline__ bool wait_stage(uint64_t* mbar, uint32_t parity) {
  bool done = false;
  const unsigned long long t_start = global_ns();
  while (!done) {
    done = mbar_done(mbar, (int)parity);
    if (!done && global_ns() - t_start > kWaitNs) break;
  }
  return __syncthreads_and(done) != 0;
}

}  // namespace cgb
