// Training passes of the warm-start network (warmstart.cuh) on the 5th-generation
// tensor cores: forward, and the backward pass of the data.
//
// A convolution is a product of 256 positions x (tap, channel) with (tap, channel) x
// 64 channels.  A layer's activations lie in shared memory as chunks of eight
// channels, 16 bytes a position, positions following each other: eight positions of a
// chunk are one 8 x 8 core matrix of a K-major operand, and a tap is a start address
// 16 bytes further on.  With 8 input channels the taps are the chunks (a distance of
// 16 bytes in K).  Two tiles of 128 positions, 64 columns of tensor memory each.
//
// Sixteen warps stage a record, and finish a layer into the next one's operand while
// a seventeenth issues the products; while those run, they write the finished layer
// to global memory.  One CTA an SM keeps the weights for all its records.
//
// What bounded the passes: mma.sync at 8 cycles an m16n8k16 and scheduler (5,100
// cycles a layer of 64 channels), its fragments read from shared memory once per 16
// positions (6,400), and the weights (94 KB) staged again for every record.  Here a
// layer takes 2,000 cycles of the tensor pipe (the instructions read their operands at
// 128 bytes a cycle); about 8,000 cycles a record with the layers' ends.  256 records:
// forward 37.2 -> 18.6 us, backward 34.6 -> 18.6; 1,024: 123 -> 52, 121 -> 61; 32
// (launch, and the weights once): 20.6 -> 12.4, 18.6 -> 12.4.
// The products are summed in the order of the fused inference's mma.sync steps (tap,
// 16 channels) and give the same bits.
#include <cuda_runtime.h>

#include <cstdint>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "warmstart.cuh"
#include "warmstart_tensor.cuh"

namespace cgb {
namespace ws {
namespace {

constexpr int kFinishers = 512;
constexpr int kConvThreads = kFinishers + 32;
constexpr int kHBytes = kNS * 128;         // one layer of one record in global memory
constexpr int kFeatBytes = kFeatRows * 16;
// Distances between chunks, odd multiples of 16 bytes: what eight lanes store for
// eight chunks falls into distinct banks.
constexpr int kActRows = 261;              // row r is position r - 2
constexpr int kActChunk = kActRows * 16, kActBytes = 8 * kActChunk;
constexpr int kWChunk = 65 * 16, kWTap = 8 * kWChunk, kWBytes = 5 * kWTap;
constexpr int kW4Chunk = 17 * 16, kW4Tap = 8 * kW4Chunk, kW4Size = 5 * kW4Tap;  // 16 outputs
static_assert(kNS + 4 <= kActRows && kNS + 5 <= kActRows, "taps stay inside");

// forward: F | A | B | W1 | W2 | W3 | W4 | bias;  backward: dO | A | B | T4 | T3 | T2
constexpr int kOffIn = 0;
constexpr int kOffA = kFeatBytes, kOffB = kOffA + kActBytes;
constexpr int kOffFirst = kOffB + kActBytes;
constexpr int kOffSecond = kOffFirst + kW1Bytes, kOffThird = kOffSecond + kWBytes;
constexpr int kOffLast = kOffThird + kWBytes, kOffBiases = kOffLast + kW4Size;
constexpr int kOffFwdShared = kOffBiases + kBiasFloats * 4;
constexpr int kOffBwdShared = kOffLast;
constexpr int kOffSquares = kOffFwdShared + (int)sizeof(TensorShared);
constexpr int kFwdBytes = kOffSquares + kNS * 8;
constexpr int kBwdBytes = kOffBwdShared + (int)sizeof(TensorShared);
static_assert(kActRows * 16 <= kFeatBytes && kOffFwdShared % 16 == 0 && kOffBwdShared % 16 == 0 &&
                  kFwdBytes <= 227 * 1024,
              "shared memory");

__device__ __forceinline__ void fill_zero(unsigned char* p) {
  *reinterpret_cast<uint4*>(p) = make_uint4(0, 0, 0, 0);
}

// A blob's 64-channel rows (row = tap * rows_tap + channel) to chunks.
__device__ __forceinline__ void stage_weights(unsigned char* dst, const unsigned char* src,
                                              int rows_tap, int chunk, int tap_bytes, int tid) {
  const int n = 5 * rows_tap * 8;
#pragma unroll 5
  for (int u = tid; u < n; u += kConvThreads) {
    const int row = u >> 3, c = (u & 7) ^ (row & 7);
    const int tap = row / rows_tap, out = row - tap * rows_tap;
    *reinterpret_cast<uint4*>(dst + tap * tap_bytes + c * chunk + out * 16) =
        __ldg(reinterpret_cast<const uint4*>(src) + u);
  }
}

// The issuing warp: products of one layer with 64 input channels, columns 64 t of
// tensor memory for tile t.
__device__ __forceinline__ void issue_conv64(TensorShared& S, uint32_t in, uint32_t w, int chunk,
                                             int tap_bytes, uint32_t ins, uint32_t tmem,
                                             uint32_t issue) {
  const uint64_t a0 = tfir::operand(in, kActChunk, 128), b0 = tfir::operand(w, chunk, 128);
#pragma unroll 1
  for (int t = 0; t < 2; ++t) {
#pragma unroll 1
    for (int tap = 0; tap < kTaps; ++tap) {
      const uint64_t a = a0 + t * 128 + tap, b = b0 + ((tap * tap_bytes) >> 4);
#pragma unroll
      for (int cb = 0; cb < 4; ++cb)
        tfir::mma(tmem + 64 * t, a + ((2 * cb * kActChunk) >> 4), b + ((2 * cb * chunk) >> 4),
                  tap > 0 || cb > 0, issue, ins);
    }
    if (issue) tfir::commit(&S.mbar[t]);
    __syncwarp();
  }
}
// And with 8; row0: the row of in that position 0 multiplies with tap 0.
__device__ __forceinline__ void issue_conv8(TensorShared& S, uint32_t in, int row0, uint32_t w,
                                            uint32_t tmem, uint32_t issue) {
  const uint64_t a = tfir::operand(in + row0 * 16, 16, 128), b = tfir::operand(w, 64 * 16, 128);
#pragma unroll
  for (int t = 0; t < 2; ++t) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
      tfir::mma(tmem + 64 * t, a + t * 128 + 2 * j, b + 2 * j * 64, j > 0, issue,
                instr(64, false));
    if (issue) tfir::commit(&S.mbar[t]);
    __syncwarp();
  }
}

// A finished layer to global memory (64-channel rows).
__device__ __forceinline__ void write_layer(unsigned char* __restrict__ dst,
                                            const unsigned char* act, int tid) {
  uint4 v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int u = tid + kFinishers * j, row = u >> 3, c = (u & 7) ^ (row & 7);
    v[j] = *reinterpret_cast<const uint4*>(act + c * kActChunk + (row + 2) * 16);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) reinterpret_cast<uint4*>(dst)[tid + kFinishers * j] = v[j];
}

// A finisher's share of a layer: position pos, channels c0 .. c0 + 31.
struct Share {
  int tile, pos, c0;
  uint32_t tmem;
  __device__ __forceinline__ Share(uint32_t base, int warp, int lane) {
    tile = (warp >> 2) & 1;
    pos = 128 * tile + 32 * (warp & 3) + lane;
    c0 = 32 * (warp >> 3);
    tmem = base + ((uint32_t)(32 * (warp & 3)) << 16) + 64 * tile + c0;
  }
  __device__ __forceinline__ void read(float (&v)[4][8]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) tfir::tmem_load8(tmem + 8 * i, v[i]);
    tfir::tmem_wait_loads();
  }
  __device__ __forceinline__ unsigned char* row(unsigned char* act) const {
    return act + (c0 >> 3) * kActChunk + (pos + 2) * 16;
  }
};

// What both kernels begin with; the address of tensor memory.
__device__ __forceinline__ uint32_t begin(unsigned char* sm, TensorShared& S, int tid, int warp) {
  if (tid == 0) init_barriers(S, kFinishers / 32);
  if (warp == kFinishers / 32) tfir::tmem_alloc(&S.tmem);
  // rows beside the positions
  if (tid < 2 * 8 * 4) {
    const int r = tid & 3, c = (tid >> 2) & 7, buf = tid >> 5;
    fill_zero(sm + (buf ? kOffB : kOffA) + c * kActChunk + (r < 2 ? r : kNS + r) * 16);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tfir::fence_before();
  __syncthreads();
  tfir::fence_after();
  return __shfl_sync(kFull, S.tmem, 0);
}

// LOSS: the loss kernel's work too (warmstart.cu), 4 us of launch and latency less.
template <bool LOSS>
__global__ void __launch_bounds__(kConvThreads, 1)
    forward_kernel(const unsigned char* __restrict__ blob, const unsigned char* __restrict__ feat,
                   int n, unsigned char* __restrict__ hid, float* __restrict__ out,
                   const float* __restrict__ target, float s_out,
                   unsigned char* __restrict__ dout, double* __restrict__ loss_part, int skip) {
  extern __shared__ __align__(128) unsigned char sm[];
  TensorShared& S = *reinterpret_cast<TensorShared*>(sm + kOffFwdShared);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* bias = reinterpret_cast<const float*>(sm + kOffBiases);
  for (int i = tid; i < kW1Bytes / 16; i += kConvThreads)
    reinterpret_cast<uint4*>(sm + kOffFirst)[i] =
        __ldg(reinterpret_cast<const uint4*>(blob + kOffW1) + i);
  if (tid < kBiasFloats * 4 / 16)
    reinterpret_cast<uint4*>(sm + kOffBiases)[tid] =
        __ldg(reinterpret_cast<const uint4*>(blob + kOffBias) + tid);
  stage_weights(sm + kOffSecond, blob + kOffW2, 64, kWChunk, kWTap, tid);
  stage_weights(sm + kOffThird, blob + kOffW3, 64, kWChunk, kWTap, tid);
  stage_weights(sm + kOffLast, blob + kOffW4, 8, kW4Chunk, kW4Tap, tid);
  for (int i = tid; i < 5 * 8 * 8; i += kConvThreads)  // outputs 8 .. 15
    fill_zero(sm + kOffLast + (i >> 3) * kW4Chunk + (8 + (i & 7)) * 16);
  const uint32_t tmem = begin(sm, S, tid, warp);
  release_next();

  if (warp == kFinishers / 32) {
    const uint32_t issue = tfir::elected(), base = tfir::saddr(sm);
    int phase = 0;
    for (int rec = blockIdx.x; rec < n; rec += gridDim.x) {
      if (!take_over(S, &S.ready[0], phase++)) break;
      if (!skip || phase > 1)
        issue_conv8(S, base + kOffIn, 6, base + kOffFirst, tmem, issue);
      if (!take_over(S, &S.ready[0], phase++)) break;
      issue_conv64(S, base + kOffA, base + kOffSecond, kWChunk, kWTap, instr(64, false), tmem, issue);
      if (!take_over(S, &S.ready[0], phase++)) break;
      issue_conv64(S, base + kOffB, base + kOffThird, kWChunk, kWTap, instr(64, false), tmem, issue);
      if (!take_over(S, &S.ready[0], phase++)) break;
      issue_conv64(S, base + kOffA, base + kOffLast, kW4Chunk, kW4Tap, instr(16, false), tmem, issue);
    }
    drain(S, issue);
  } else {
    const Share mine(tmem, warp, lane);
    int phase = 0;
    uint4 next = make_uint4(0, 0, 0, 0);
    auto load = [&](int rec) {
      if (tid < kFeatRows)
        next = __ldg(reinterpret_cast<const uint4*>(feat + (int64_t)rec * kFeatBytes) + tid);
    };
    // bias, ReLU, BF16: a hidden layer into the next operand
    auto hidden = [&](unsigned char* act, const float* b) {
      wait_products(S, mine.tile, phase++);
      tfir::fence_after();
      float v[4][8];
      mine.read(v);
      unsigned char* dst = mine.row(act);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float r[8];
#pragma unroll
        for (int c = 0; c < 8; c += 4) {
          const float4 q = *reinterpret_cast<const float4*>(b + mine.c0 + 8 * i + c);
          r[c] = fmaxf(v[i][c] + q.x, 0.0f);
          r[c + 1] = fmaxf(v[i][c + 1] + q.y, 0.0f);
          r[c + 2] = fmaxf(v[i][c + 2] + q.z, 0.0f);
          r[c + 3] = fmaxf(v[i][c + 3] + q.w, 0.0f);
        }
        *reinterpret_cast<uint4*>(dst + i * kActChunk) =
            make_uint4(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]), pack_bf16(r[4], r[5]),
                       pack_bf16(r[6], r[7]));
      }
      hand_over(S, 0, lane);
      // what is copied next was written by all
      asm volatile("bar.sync 2, %0;" ::"n"(kFinishers) : "memory");
    };
    if (blockIdx.x < n) load(blockIdx.x);
    for (int rec = blockIdx.x; rec < n; rec += gridDim.x) {
      unsigned char* h = hid + (int64_t)rec * kHBytes;
      if (tid < kFeatRows) reinterpret_cast<uint4*>(sm + kOffIn)[tid] = next;
      hand_over(S, 0, lane);
      if (rec + gridDim.x < n) load(rec + gridDim.x);
      hidden(sm + kOffA, bias);
      write_layer(h, sm + kOffA, tid);
      hidden(sm + kOffB, bias + 64);
      write_layer(h + (int64_t)n * kHBytes, sm + kOffB, tid);
      hidden(sm + kOffA, bias + 128);
      write_layer(h + 2 * (int64_t)n * kHBytes, sm + kOffA, tid);
      wait_products(S, mine.tile, phase++);
      tfir::fence_after();
      if (mine.c0 == 0) {
        float v[8];
        tfir::tmem_load8(mine.tmem, v);
        tfir::tmem_wait_loads();
        const bool failed = *(volatile int*)&S.failed;
        const float o = failed ? __int_as_float(0x7fffffff) : v[0] + bias[192];
        out[(int64_t)rec * kNS + mine.pos] = o;
        if (LOSS) {
          double* red = reinterpret_cast<double*>(sm + kOffSquares);
          const float e = s_out * o - target[(int64_t)rec * kNS + mine.pos];
          const float gsc = 2.0f * s_out / ((float)n * 256.0f);
          reinterpret_cast<uint4*>(dout)[(int64_t)rec * kNS + mine.pos] =
              make_uint4(failed ? 0x7fffu : bf16_bits(gsc * e), 0, 0, 0);
          red[mine.pos] = (double)e * (double)e;
          // (warps 0 to 7; the next record's squares come after barriers of all)
          asm volatile("bar.sync 3, %0;" ::"n"(kNS) : "memory");
          if (warp == 0) {
            double r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = red[lane + 32 * i] + red[lane + 32 * i + 128];
            r[0] += r[2];
            r[1] += r[3];
            r[0] += r[1];
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) r[0] += __shfl_down_sync(kFull, r[0], o);
            if (lane == 0) loss_part[rec] = r[0];
          }
        }
      }
    }
    tfir::fence_before();
  }
  __syncthreads();
  if (warp == kFinishers / 32) tfir::tmem_free(tmem);
}

// dH3 = (W4^T * dO) . [H3 > 0], dH2 = (W3^T * dH3) . [H2 > 0],
// dH1 = (W2^T * dH2) . [H1 > 0], with the transposed, tap-reversed weights.
__global__ void __launch_bounds__(kConvThreads, 1)
    backward_kernel(const unsigned char* __restrict__ blobT,
                    const unsigned char* dout, const unsigned char* hid, int n,
                    unsigned char* dpre, int skip) {
  extern __shared__ __align__(128) unsigned char sm[];
  TensorShared& S = *reinterpret_cast<TensorShared*>(sm + kOffBwdShared);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kW1Bytes / 16; i += kConvThreads)
    reinterpret_cast<uint4*>(sm + kOffFirst)[i] =
        __ldg(reinterpret_cast<const uint4*>(blobT + kOffT4) + i);
  stage_weights(sm + kOffSecond, blobT + kOffT3, 64, kWChunk, kWTap, tid);
  stage_weights(sm + kOffThird, blobT + kOffT2, 64, kWChunk, kWTap, tid);
  if (tid < kActRows - kNS) fill_zero(sm + kOffIn + (tid < 2 ? tid : kNS + tid) * 16);
  const uint32_t tmem = begin(sm, S, tid, warp);
  release_next();
  wait_previous(dout, hid);

  if (warp == kFinishers / 32) {
    const uint32_t issue = tfir::elected(), base = tfir::saddr(sm);
    int phase = 0;
    for (int rec = blockIdx.x; rec < n; rec += gridDim.x) {
      if (!take_over(S, &S.ready[0], phase++)) break;
      if (!skip || phase > 1)
        issue_conv8(S, base + kOffIn, 0, base + kOffFirst, tmem, issue);
      if (!take_over(S, &S.ready[0], phase++)) break;
      issue_conv64(S, base + kOffA, base + kOffSecond, kWChunk, kWTap, instr(64, false), tmem, issue);
      if (!take_over(S, &S.ready[0], phase++)) break;
      issue_conv64(S, base + kOffB, base + kOffThird, kWChunk, kWTap, instr(64, false), tmem, issue);
    }
    drain(S, issue);
  } else {
    const Share mine(tmem, warp, lane);
    int phase = 0;
    uint4 next = make_uint4(0, 0, 0, 0), mask[4];
    auto load = [&](int rec) {
      if (tid < kNS) next = load_written(reinterpret_cast<const uint4*>(dout) + (int64_t)rec * kNS + tid);
    };
    // the activations that mask this thread's share of a layer
    auto load_mask = [&](int rec, int layer) {
      const uint4* src = reinterpret_cast<const uint4*>(hid + ((int64_t)layer * n + rec) * kHBytes);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        mask[i] = load_written(src + mine.pos * 8 + (((mine.c0 >> 3) + i) ^ (mine.pos & 7)));
    };
    auto masked = [&](unsigned char* act) {
      wait_products(S, mine.tile, phase++);
      tfir::fence_after();
      float v[4][8];
      mine.read(v);
      unsigned char* dst = mine.row(act);
      const bool failed = *(volatile int*)&S.failed;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t m[4] = {mask[i].x, mask[i].y, mask[i].z, mask[i].w};
        uint32_t w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          w[c] = pack_bf16(bf16_lo(m[c]) > 0.0f ? v[i][2 * c] : 0.0f,
                           bf16_hi(m[c]) > 0.0f ? v[i][2 * c + 1] : 0.0f);
          if (failed) w[c] = 0x7fff7fffu;
        }
        *reinterpret_cast<uint4*>(dst + i * kActChunk) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    };
    if (blockIdx.x < n) load(blockIdx.x);
    for (int rec = blockIdx.x; rec < n; rec += gridDim.x) {
      unsigned char* d = dpre + (int64_t)rec * kHBytes;
      if (tid < kNS) reinterpret_cast<uint4*>(sm + kOffIn)[tid + 2] = next;
      hand_over(S, 0, lane);
      load_mask(rec, 2);
      if (rec + gridDim.x < n) load(rec + gridDim.x);
      masked(sm + kOffA);
      hand_over(S, 0, lane);
      load_mask(rec, 1);
      asm volatile("bar.sync 2, %0;" ::"n"(kFinishers) : "memory");
      write_layer(d + 2 * (int64_t)n * kHBytes, sm + kOffA, tid);
      masked(sm + kOffB);
      hand_over(S, 0, lane);
      load_mask(rec, 0);
      asm volatile("bar.sync 2, %0;" ::"n"(kFinishers) : "memory");
      write_layer(d + (int64_t)n * kHBytes, sm + kOffB, tid);
      masked(sm + kOffA);
      asm volatile("bar.sync 2, %0;" ::"n"(kFinishers) : "memory");
      write_layer(d, sm + kOffA, tid);
    }
    tfir::fence_before();
  }
  __syncthreads();
  if (warp == kFinishers / 32) tfir::tmem_free(tmem);
}

// One CTA fits an SM.
int conv_grid(int n, int* grid) {
  int dev = 0, sms = 0;
  CGB_TRY_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
  CGB_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev),
               "cudaDeviceGetAttribute");
  *grid = n < sms ? n : sms;
  return CGB_OK;
}

}  // namespace
}  // namespace ws
}  // namespace cgb

using namespace cgb;
using namespace cgb::ws;

int cgb::ws::g_fault_skip_products = 0;

extern "C" int cgb_ws_set_fault_injection(int skip_products) {
  g_fault_skip_products = skip_products ? 1 : 0;
  return CGB_OK;
}

template <bool LOSS>
static int launch_forward(const void* d_blob, const void* d_feat, int n, void* d_hid, float* d_out,
                          const float* d_target, float s_out, void* d_dout, double* d_loss_part,
                          void* stream) {
  int grid = 0;
  if (const int rc = conv_grid(n, &grid)) return rc;
  CGB_TRY_CUDA(cudaFuncSetAttribute(forward_kernel<LOSS>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdBytes),
               "cudaFuncSetAttribute(forward)");
  forward_kernel<LOSS><<<grid, kConvThreads, kFwdBytes, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const unsigned char*>(d_blob), static_cast<const unsigned char*>(d_feat), n,
      static_cast<unsigned char*>(d_hid), d_out, d_target, s_out,
      static_cast<unsigned char*>(d_dout), d_loss_part, g_fault_skip_products);
  CGB_TRY_CUDA(cudaGetLastError(), "forward_kernel launch");
  note_launch();
  return CGB_OK;
}

extern "C" int cgb_ws_forward_dev(const void* d_blob, const void* d_feat, int n, void* d_hid,
                                  float* d_out, void* stream) {
  if (n == 0) return CGB_OK;
  if (n < 0 || !d_blob || !d_feat || !d_hid || !d_out)
    return fail(CGB_ERR_ARG, "cgb_ws_forward_dev: bad arguments");
  return launch_forward<false>(d_blob, d_feat, n, d_hid, d_out, nullptr, 0.0f, nullptr, nullptr,
                               stream);
}

int cgb::ws::forward_loss(const void* d_blob, const void* d_feat, int n, void* d_hid, float* d_out,
                          const float* d_target, float s_out, void* d_dout, double* d_loss_part,
                          void* stream) {
  if (n == 0) return CGB_OK;
  if (n < 0 || !d_blob || !d_feat || !d_hid || !d_out)
    return fail(CGB_ERR_ARG, "cgb_ws_forward_dev: bad arguments");
  if (!d_target || !d_dout || !d_loss_part)
    return fail(CGB_ERR_ARG, "cgb_ws_loss_dev: bad arguments");
  return launch_forward<true>(d_blob, d_feat, n, d_hid, d_out, d_target, s_out, d_dout, d_loss_part,
                              stream);
}

static int launch_backward(bool after, const void* d_blobT, const void* d_dout, const void* d_hid,
                           int n, void* d_dpre, void* stream) {
  if (n == 0) return CGB_OK;
  if (n < 0 || !d_blobT || !d_dout || !d_hid || !d_dpre)
    return fail(CGB_ERR_ARG, "cgb_ws_backward_dev: bad arguments");
  int grid = 0;
  if (const int rc = conv_grid(n, &grid)) return rc;
  CGB_TRY_CUDA(cudaFuncSetAttribute(backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kBwdBytes),
               "cudaFuncSetAttribute(backward)");
  CGB_TRY_CUDA(launch_after(after, backward_kernel, grid, kConvThreads, kBwdBytes,
                            reinterpret_cast<cudaStream_t>(stream),
                            static_cast<const unsigned char*>(d_blobT),
                            static_cast<const unsigned char*>(d_dout),
                            static_cast<const unsigned char*>(d_hid), n,
                            static_cast<unsigned char*>(d_dpre), g_fault_skip_products),
               "backward_kernel launch");
  note_launch();
  return CGB_OK;
}

extern "C" int cgb_ws_backward_dev(const void* d_blobT, const void* d_dout, const void* d_hid,
                                   int n, void* d_dpre, void* stream) {
  return launch_backward(false, d_blobT, d_dout, d_hid, n, d_dpre, stream);
}

int cgb::ws::backward_after(const void* d_blobT, const void* d_dout, const void* d_hid, int n,
                            void* d_dpre, void* stream) {
  return launch_backward(true, d_blobT, d_dout, d_hid, n, d_dpre, stream);
}
