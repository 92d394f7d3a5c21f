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
  uint64_t mbar[3];   // the products of tile (or accumulator) h are done
  uint64_t ready[2];  // the operands (of stage h) are in shared memory: an arrival a warp
  uint64_t drained;   // all products that were issued are done
  uint32_t tmem;
  int failed;         // a wait ran out
};

// FP32 accumulators, BF16 operands (both K-major, or both MN-major), M = 128.
__host__ __device__ constexpr uint32_t instr(int n, bool mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? 3u << 15 : 0u) |
         ((uint32_t)(n / 8) << 17) | (8u << 24);
}

// warps: that prepare the operands
__device__ __forceinline__ void init_barriers(TensorShared& S, int warps) {  // one thread
  for (int h = 0; h < 3; ++h) mbar_init(&S.mbar[h], 1);
  for (int h = 0; h < 2; ++h) mbar_init(&S.ready[h], warps);
  mbar_init(&S.drained, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  S.failed = 0;
}

// Completion `phase` (from 0) of mbar[h].  Bounded; after a wait that ran out none
// waits, and the kernel's results become NaN.
__device__ __forceinline__ void wait_products(TensorShared& S, int h, int phase) {
  unsigned long long start = 0;
  while (!mbar_done(&S.mbar[h], phase)) {
    if (*(volatile int*)&S.failed) break;
    if (start == 0) start = global_ns();
    if (global_ns() - start > kWaitNs) *(volatile int*)&S.failed = 1;
  }
}

// This warp's share of an operand (of stage h) is in shared memory.
__device__ __forceinline__ void hand_over(TensorShared& S, int h, int lane) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tfir::fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(&S.ready[h]);
}
// The issuing warp, converged: completion `phase` of a barrier that the other warps
// arrive at; false after a wait that ran out.
__device__ __forceinline__ bool take_over(TensorShared& S, uint64_t* bar, int phase) {
  const unsigned long long start = global_ns();
  while (!__all_sync(kFull, mbar_done(bar, phase))) {
    // (the other warps' work between two operands is far shorter, their waits a fourth)
    const bool late = global_ns() - start > 4 * kWaitNs;
    if (__any_sync(kFull, late || *(volatile int*)&S.failed)) return false;
  }
  tfir::fence_after();
  return true;
}
// The issuing warp's last step: the shared memory that its products read and the
// tensor memory that they write are given up only after the last of them, also where
// nobody waited for it.
__device__ __forceinline__ void drain(TensorShared& S, uint32_t issue) {
  if (issue) tfir::commit(&S.drained);
  const unsigned long long start = global_ns();
  while (!mbar_done(&S.drained, 0) && global_ns() - start < kWaitNs) {
  }
  __syncwarp();
}

// Test-only (cgb_ws_set_fault_injection): the next launches leave out products that
// are waited for.
extern int g_fault_skip_products;

// A training step's kernels are launched so that one's CTAs start where the one
// before it leaves an SM (launch_after): weights, zero rows and tensor memory are
// prepared beside its last records, and the launch takes no time of its own.
// release_next() comes after the CTA's own tensor memory is allocated, so that a CTA
// which holds tensor memory only ever waits for CTAs that have theirs.
// wait_previous() comes before the first access to what the earlier kernels write,
// whose addresses it passes on: the compiler may move load_written, but not over the
// wait (with plain loads 2 us more at 256 records).  wgrad releases its sum's CTAs only
// by ending: started early they cost it 2 to 3 us.  Measured (GB300), step of 32 / 256 /
// 1,024 records: 41.0 / 61.5 / 183 -> 32.8 / 55.3 / 174 us.
__device__ __forceinline__ void release_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... T>
__device__ __forceinline__ void wait_previous(const T*&... written) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  ((void)[](const T*& p) { asm volatile("" : "+l"(p)::"memory"); }(written), ...);
}

__device__ __forceinline__ uint4 load_written(const uint4* p) {
  uint4 v;
  asm("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p));
  return v;
}

// after: the kernel before it on the stream is the step's previous one.
template <typename... Params, typename... Args>
cudaError_t launch_after(bool after, void (*kernel)(Params...), int grid, int threads, int smem,
                         cudaStream_t st, Args... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3((unsigned)grid);
  config.blockDim = dim3((unsigned)threads);
  config.dynamicSmemBytes = (size_t)smem;
  config.stream = st;
  config.attrs = &attr;
  config.numAttrs = after ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// cgb_ws_backward_dev, after the forward pass of the same step (warmstart_conv.cu).
int backward_after(const void* d_blobT, const void* d_dout, const void* d_hid, int n, void* d_dpre,
                   void* stream);

}  // namespace ws
}  // namespace cgb
