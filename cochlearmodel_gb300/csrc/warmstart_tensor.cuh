// What the warm-start network's tensor-core kernels share: the instruction's
// descriptor, their barriers and a bounded wait.
#pragma once

#include "ihc_common.cuh"
#include "tensor_fir.cuh"

namespace cgb {
namespace ws {

// cgb_ws_forward_dev and cgb_ws_loss_dev in one kernel (warmstart_conv.cu).
int forward_loss(const void* d_blob, const void* d_feat, int n, void* d_hid, float* d_out,
                 const float* d_target, float s_out, void* d_dout, double* d_loss_part,
                 void* stream);

struct TensorShared {
  uint64_t mbar[2];  // the products of stage (or tile) h are done
  uint32_t tmem;
  int failed;        // a wait ran out
};

// FP32 accumulators, BF16 operands (both K-major, or both MN-major), M = 128.
__host__ __device__ constexpr uint32_t instr(int n, bool mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? 3u << 15 : 0u) |
         ((uint32_t)(n / 8) << 17) | (8u << 24);
}

__device__ __forceinline__ void init_barriers(TensorShared& S) {  // one thread
  for (int h = 0; h < 2; ++h)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tfir::saddr(&S.mbar[h])));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  S.failed = 0;
}

// Completion `phase` (from 0) of mbar[h].  Bounded; after a wait that ran out none
// waits, and the kernel's results become NaN.
__device__ __forceinline__ void wait_products(TensorShared& S, int h, int phase) {
  uint32_t done = 0;
  unsigned long long start = 0;
  while (!done) {
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(tfir::saddr(&S.mbar[h])), "r"((uint32_t)(phase & 1))
        : "memory");
    if (done || *(volatile int*)&S.failed) break;
    if (start == 0) start = global_ns();
    if (global_ns() - start > kWaitNs) *(volatile int*)&S.failed = 1;
  }
}

}  // namespace ws
}  // namespace cgb
