// Weight gradients of the warm-start network (warmstart.cuh) on the
// 5th-generation tensor cores.
//
//   dW_l[tap][co][ci] = sum over records and positions of
//                       dPre_l[pos][co] * In_l[pos + tap - 2][ci]
// is a product whose K dimension is the position.  Both factors lie in shared
// memory as they are in global memory, eight channels of a position in 16 bytes,
// the rows of one chunk of eight channels following each other: eight positions
// of a chunk are one 8 x 8 core matrix of an MN-major operand, and a shift by one
// position (a tap) is a start address 16 bytes further on.
//   layers 2, 3: M = 128 is dPre's 64 channels twice, the second time one position
//                on, N = 64 input channels: one instruction gives two taps, three
//                (at shifts -1, 1, 2 of the input) all five.
//   layers 1, 4: the operand with 8 channels is A, and its 16 chunks of eight rows
//                of M are the same rows from 16 positions on (a stride of 16 bytes),
//                of which five are the taps.
// Rows of ones beside an operand give the bias gradients in the same way.
//
// A third of the CTAs takes layer 2, layer 3, and layers 1 and 4 each, about equal
// shares of the tensor pipe (2,500 cycles a record: the instructions read their
// operands from shared memory, 49 cycles for 128 x 64 x 16).  A CTA stages a record
// while the one before is multiplied.  A record's products have sums of their own, which
// are added to the slot's as FP32 pairs by TwoSum, their high parts in registers, their
// low parts in tensor memory: one accumulator is added while the next is multiplied, so
// the adding takes no time of its own.  (In one accumulator over all of a slot's records each of
// their steps is rounded, or cut: 2,560 records of one sign 2^-14 off, 300 in one slot
// 2^-11, now 2^-18 as one record.)  A CTA writes its slot once, the low parts where there is
// room (a slot of one record has none); the slots are added in a fixed order
// (deterministic).
//
// What bounded it: with mma.sync a CTA per record staged the factors of all layers
// (209 KB), had 65 small tasks for eight warps, and added each to its slot in global
// memory.  256 records 160 -> 29 us, 1,024 records 390 -> 75, 32 records 52 -> 12 (both
// kernels).  Setting up all of shared memory and writing the slots from the accumulators'
// lanes (256 bytes apart) cost 12 us of 35.  Records in one accumulator, the slots' sums
// rounded: 17, 51 and 11.5 us; staged by cp.async instead of through registers, which
// leaves a record's trip from L2 one record's products to hide under: 37, 89 and 15.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "warmstart.cuh"
#include "warmstart_tensor.cuh"

namespace cgb {
namespace ws {
namespace {

constexpr int kLoaders = 512;                 // threads that stage the factors
constexpr int kGradThreads = kLoaders + 128;  // and the issuing warp's group of four
// registers a thread: 96 at launch, then 112 for the loaders (the sums' high parts and
// the next record) and 32 for the issuing warp's group, together the same
constexpr int kLoaderRegs = 112, kIssueRegs = 32;
static_assert(kLoaders * kLoaderRegs + 128 * kIssueRegs <= kGradThreads * 96, "register split");
constexpr int kGroups = 3;                    // layer 2 | layer 3 | layers 1 and 4

// Layers 2, 3.  K runs over positions -1 .. 270 (17 steps); row r of A's first
// half is position r - 1, of its second half r, of B r - 2.  The distances between
// chunks are odd multiples of 16 bytes: the eight chunks of a position, stored by
// eight lanes, fall into distinct banks.
constexpr int kSteps = 17;
constexpr int kARows = 273, kBRows = 275;
constexpr int kAChunk = kARows * 16, kBChunk = kBRows * 16;
constexpr int kOffB = 16 * kAChunk;           // A: 16 chunks
constexpr int kStage23 = kOffB + 10 * kBChunk;  // B: 8 chunks and two of ones
// Layers 1, 4.  K runs over positions 0 .. 255; row r of the features is position
// r - 8, of dO r - 2, of dPre and H3 r.
constexpr int kORows = 272, kHRows = 257;
constexpr int kHChunk = kHRows * 16;
constexpr int kFeat = kFeatRows * 16;
constexpr int kOffO = kFeat, kOffD = kOffO + kORows * 16, kOffH = kOffD + 8 * kHChunk;
constexpr int kStage14 = kOffH + 10 * kHChunk;  // H3: 8 chunks and two of ones
constexpr int kStage = kStage23 > kStage14 ? kStage23 : kStage14;
// the last row that a core matrix of the shifted operands reads
static_assert(6 + 240 + 15 + 15 < kFeatRows && 240 + 15 + 15 < kORows, "shifts stay inside");
static_assert(16 * kSteps <= kARows && 3 + 16 * kSteps <= kBRows && 256 <= kHRows &&
                  16 + 16 <= kHRows, "steps stay inside");

struct GradShared : TensorShared {
  uint64_t taken[3];  // accumulator j has been read: an arrival a warp
};
constexpr int kGradSmem = 2 * kStage + (int)sizeof(GradShared);
static_assert(kStage % 16 == 0 && kGradSmem <= 227 * 1024, "stages");

// MN-major operand without swizzle: distances of the core matrices that follow
// each other in K (always the next eight rows) and in M or N.
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t mn_bytes) {
  return tfir::operand(addr, 128, mn_bytes);
}
// accumulator columns: layers 2 and 3 shifts -1, 1, 2, layers 1 and 4 W1, b1, W4; the
// products with ones (a column of b2, b3, b4) behind the first, or the last
__device__ __forceinline__ int acc_column(bool ends, int j) {  // ends: layers 1 and 4
  return 64 * j + (!ends && j > 0 ? 32 : 0);
}
__device__ __forceinline__ int ones_column(bool ends) { return ends ? 192 : 64; }
constexpr int kLow = 256;  // the slot's low parts, accumulator j from 64 j on
static_assert(kLow + 3 * 64 <= (int)tfir::kTmemCols, "tensor memory");

__global__ void __launch_bounds__(kGradThreads, 1)
    wgrad_kernel(const unsigned char* __restrict__ feat, const unsigned char* hid,
                 const unsigned char* dpre, const unsigned char* dout, int n, int parts,
                 int lows, float* partial, int skip) {
  extern __shared__ __align__(128) unsigned char sm[];
  GradShared& S = *reinterpret_cast<GradShared*>(sm + 2 * kStage);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = blockIdx.x % kGroups, slot = blockIdx.x / kGroups;
  if (tid == 0) {
    for (int j = 0; j < 3; ++j) mbar_init(&S.taken[j], kLoaders / 32);
    init_barriers(S, kLoaders / 32);
  }
  if (warp == kLoaders / 32) tfir::tmem_alloc(&S.tmem);
  // zero rows around the positions, and the rows of ones
  for (int st = 0; st < 2; ++st) {
    unsigned char* s = sm + st * kStage;
    auto fill = [&](int off, uint32_t w) {
      *reinterpret_cast<uint4*>(s + off) = make_uint4(w, w, w, w);
    };
    if (group < 2) {
      for (int i = tid; i < 16 * 16; i += kGradThreads) {
        const int c = i >> 4, r = i & 15;
        fill(c * kAChunk + (c < 8 && r == 0 ? 0 : 256 + r) * 16, 0);
      }
      constexpr int kEdge = kBRows - kNS;
      for (int i = tid; i < 8 * kEdge; i += kGradThreads) {
        const int c = i / kEdge, r = i - c * kEdge;
        fill(kOffB + c * kBChunk + (r < 2 ? r : kNS + r) * 16, 0);
      }
      for (int i = tid; i < 2 * kBRows; i += kGradThreads)
        fill(kOffB + 8 * kBChunk + i * 16, 0x3f803f80u);
    } else {
      if (tid < kORows - kNS) fill(kOffO + (tid < 2 ? tid : kNS + tid) * 16, 0);
      for (int i = tid; i < 2 * kHRows; i += kGradThreads)
        fill(kOffH + 8 * kHChunk + i * 16, 0x3f803f80u);
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tfir::fence_before();
  __syncthreads();
  tfir::fence_after();
  const uint32_t tmem = __shfl_sync(kFull, S.tmem, 0);
  wait_previous(hid, dpre, dout);
  const int64_t layer = (int64_t)n * kNS * 128;  // bytes of a layer of hid, dpre
  const int records = slot < n ? (n - slot + parts - 1) / parts : 0;

  if (warp >= kLoaders / 32)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
  if (warp == kLoaders / 32) {
    const uint32_t issue = tfir::elected();
    for (int it = 0; it < records; ++it) {
      const int st = it & 1;
      const uint32_t base = tfir::saddr(sm) + st * kStage;
      if (!take_over(S, &S.ready[st], it >> 1)) break;
      if (skip) continue;
      const uint64_t a = operand(base, kAChunk), b = operand(base + kOffB, kBChunk);
      const uint64_t f = operand(base + 6 * 16, 16), o = operand(base + kOffO, 16),
                     ones = operand(base + kOffH + 8 * kHChunk, 16),
                     d = operand(base + kOffD, kHChunk), h = operand(base + kOffH, kHChunk);
      bool ok = true;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (it > 0 && !take_over(S, &S.taken[j], it - 1)) {
          ok = false;
          break;
        }
        const uint32_t acc = tmem + acc_column(group == 2, j);
        if (group < 2) {
#pragma unroll 1
          for (int k = 0; k < kSteps; ++k)  // 16 rows of 16 bytes
            tfir::mma(acc, a + 16 * k, b + 16 * k + (j == 0 ? 0 : j + 1), k > 0, issue,
                      instr(j == 0 ? 80 : 64, true));
        } else {
#pragma unroll 1
          for (int k = 0; k < kNS / 16; ++k)
            tfir::mma(acc, (j == 0 ? f : j == 1 ? ones : o) + 16 * k, (j == 2 ? h : d) + 16 * k,
                      k > 0, issue, instr(j == 2 ? 80 : 64, true));
        }
        if (issue) tfir::commit(&S.mbar[j]);
        __syncwarp();
      }
      if (!ok) break;
    }
    drain(S, issue);
  } else if (warp < kLoaders / 32) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kLoaderRegs));
    auto run = [&](auto ends) {
    constexpr bool kEnds = decltype(ends)::value;  // layers 1 and 4
    // 16 bytes u of a record: row u / 8, and its chunk by the rows' swizzle.  The
    // first factor (dPre) in g[0..3], the second (In) in g[4..7]; layers 1 and 4
    // have the features and dO in g[8], g[9].
    const unsigned char* first = dpre + (kEnds ? 0 : (group + 1) * layer);
    const unsigned char* second = hid + (kEnds ? 2 : group) * layer;
    uint4 g[kEnds ? 10 : 8];
    auto load = [&](int rec) {
      const uint4* p = reinterpret_cast<const uint4*>(first + (int64_t)rec * kNS * 128);
      const uint4* q = reinterpret_cast<const uint4*>(second + (int64_t)rec * kNS * 128);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        g[j] = load_written(p + tid + kLoaders * j);
        g[4 + j] = load_written(q + tid + kLoaders * j);
      }
      if constexpr (kEnds) {
        if (tid < kFeatRows)
          g[8] = __ldg(reinterpret_cast<const uint4*>(feat + (int64_t)rec * kFeat) + tid);
        if (tid < kNS)
          g[9] = load_written(reinterpret_cast<const uint4*>(dout + (int64_t)rec * kNS * 16) + tid);
      }
    };
    auto store = [&](int st) {
      unsigned char* s = sm + st * kStage;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int u = tid + kLoaders * j, row = u >> 3, c = (u & 7) ^ (row & 7);
        if constexpr (!kEnds) {
          *reinterpret_cast<uint4*>(s + c * kAChunk + (row + 1) * 16) = g[j];
          *reinterpret_cast<uint4*>(s + (8 + c) * kAChunk + row * 16) = g[j];
          *reinterpret_cast<uint4*>(s + kOffB + c * kBChunk + (row + 2) * 16) = g[4 + j];
        } else {
          *reinterpret_cast<uint4*>(s + kOffD + c * kHChunk + row * 16) = g[j];
          *reinterpret_cast<uint4*>(s + kOffH + c * kHChunk + row * 16) = g[4 + j];
        }
      }
      if constexpr (kEnds) {
        if (tid < kFeatRows) *reinterpret_cast<uint4*>(s + tid * 16) = g[8];
        if (tid < kNS) *reinterpret_cast<uint4*>(s + kOffO + (tid + 2) * 16) = g[9];
      }
      hand_over(S, st, lane);
    };
    // lane = row of M, sixteen columns of an accumulator a warp
    const int quarter = warp & 3, m = 32 * quarter + lane, c0 = (warp >> 2) * 16;
    const uint32_t lanes = tmem + ((uint32_t)(32 * quarter) << 16);
    // of layers 1 and 4 the rows past the taps' 40 are nothing
    const bool rows = !kEnds || quarter < 2;
    float hi[3][16], hi1 = 0.0f, lo1 = 0.0f;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int c = 0; c < 16; ++c) hi[j][c] = 0.0f;
    // accumulator j of record it to the slot's sums
    auto add = [&](int j, int it) {
      if (rows) {
        const uint32_t acc = lanes + acc_column(kEnds, j) + c0, low = lanes + kLow + 64 * j + c0;
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
          float v[4], lo[4];
          tfir::tmem_load4(acc + c, v);
          tfir::tmem_load4(low + c, lo);
          tfir::tmem_wait_loads();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (it == 0) lo[i] = 0.0f;
            two_sum_add(hi[j][c + i], lo[i], v[i]);
          }
          tfir::tmem_store4(low + c, lo);
        }
        if (c0 == 0 && j == (kEnds ? 2 : 0)) {
          float v[8];
          tfir::tmem_load8(lanes + ones_column(kEnds), v);
          tfir::tmem_wait_loads();
          two_sum_add(hi1, lo1, v[0]);
        }
        tfir::tmem_wait_stores();
      }
      tfir::fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.taken[j]);
    };
    if (records) load(slot);
#pragma unroll 1
    for (int it = 0; it <= records; ++it) {
      // (the products of record it - 2, of the same stage, have been added)
      if (it < records) store(it & 1);
      if (it + 1 < records) load(slot + (it + 1) * parts);
      if (it == 0) continue;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        wait_products(S, j, it - 1);
        tfir::fence_after();
        add(j, it - 1);
      }
    }

    // The group's part of the slot, put together in shared memory (the products have been
    // read); the low parts, if they have a row, in a second round.
    const bool failed = *(volatile int*)&S.failed, split = slot < lows;
    float* const out = reinterpret_cast<float*>(sm);
    auto put = [](float* dst, const float (&v)[8]) {
#pragma unroll
      for (int i = 0; i < 8; ++i) dst[i] = v[i];
    };
#pragma unroll 1
    for (int low = 0; low < (split ? 2 : 1); ++low) {
      asm volatile("bar.sync 3, %0;" ::"n"(kLoaders) : "memory");
      // columns c0 + c .. + 7 of accumulator j, and the column of ones
      // (a sum out of FP32's range has no low part)
      auto value = [&](float h, float l) {
        l = fabsf(h) < __int_as_float(0x7f800000) ? l : 0.0f;
        return failed ? __int_as_float(0x7fffffff) : low ? l : split ? h : __fadd_rn(h, l);
      };
      auto read = [&](int j, int c, float (&v)[8]) {
        float lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) lo[i] = 0.0f;
        if (records) {
          tfir::tmem_load8(lanes + kLow + 64 * j + c0 + c, lo);
          tfir::tmem_wait_loads();
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = value(hi[j][c + i], lo[i]);
      };
      const float v1 = value(hi1, lo1);
      float* part = partial + (int64_t)(low ? parts + slot : slot) * kParams;
      float v[8];
      if constexpr (!kEnds) {
        constexpr int kPitch = 65;  // [tap][co] rows of 64 ci, then the bias gradients
        const int half = m >> 6, co = m & 63;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int tap = (j == 0 ? 1 : j + 2) - half;
#pragma unroll
          for (int c = 0; c < 16; c += 8) {
            read(j, c, v);
            if (!(j == 2 && half)) put(out + (tap * 64 + co) * kPitch + c0 + c, v);
          }
        }
        if (c0 == 0 && !half) out[co * kPitch + 64] = v1;
        asm volatile("bar.sync 3, %0;" ::"n"(kLoaders) : "memory");
        static_assert(ob2 == oW2 + 5 * 64 * 64 && ob3 == oW3 + 5 * 64 * 64, "bias after weights");
        float* W = part + (group ? oW3 : oW2);
#pragma unroll 8
        for (int i = tid; i < 5 * 64 * 64; i += kLoaders) W[i] = out[(i >> 6) * kPitch + (i & 63)];
        if (tid < 64) W[5 * 64 * 64 + tid] = out[tid * kPitch + 64];
      } else {
        constexpr int kPitch = 9;  // [tap][co] rows of 8 ci; b1; W4, b4
        float* const out4 = out + 5 * 64 * kPitch + 64;
        if (rows) {
#pragma unroll
          for (int c = 0; c < 16; c += 8) {
            read(0, c, v);
            if (m < 40)
#pragma unroll
              for (int i = 0; i < 8; ++i)
                out[((m >> 3) * 64 + c0 + c + i) * kPitch + (m & 7)] = v[i];
            read(1, c, v);
            if (m == 0) put(out + 5 * 64 * kPitch + c0 + c, v);
            read(2, c, v);
            if (m < 40 && (m & 7) == 0) put(out4 + (4 - (m >> 3)) * 64 + c0 + c, v);
          }
          if (c0 == 0 && m == 16) out4[5 * 64] = v1;
        }
        asm volatile("bar.sync 3, %0;" ::"n"(kLoaders) : "memory");
        static_assert(ob1 == oW1 + 5 * 64 * 8 && ob4 == oW4 + 5 * 64, "bias after weights");
        for (int i = tid; i < 5 * 64 * 8; i += kLoaders)
          part[oW1 + i] = out[(i >> 3) * kPitch + (i & 7)];
        if (tid < 64) part[ob1 + tid] = out[5 * 64 * kPitch + tid];
        if (tid < 5 * 64 + 1) part[oW4 + tid] = out4[tid];
      }
    }
    };
    if (group < 2)
      run(std::false_type());
    else
      run(std::true_type());
    tfir::fence_before();
  }
  __syncthreads();
  if (warp == kLoaders / 32) tfir::tmem_free(tmem);
}

// Sum over the slots in order, as an unevaluated sum of three FP32 values, the errors of
// the rounded sum's errors kept too: within n^3 2^-72 of the magnitudes, an FP64 sum's
// n 2^-53 for the 100 rows there are (which at a 64th of FP32's rate would take 8 us); a
// sum that leaves the FP32 range on the way is taken in FP64.  The last CTA, if there is a
// loss to be given, takes the records' losses instead.
constexpr int kSumThreads = 128;

__global__ void __launch_bounds__(kSumThreads)
    reduce_kernel(const float* partial, int parts, float* __restrict__ grad,
                  const double* loss_part, int n, double* __restrict__ loss) {
  wait_previous(partial, loss_part);
  if (loss && blockIdx.x == gridDim.x - 1) {
    __shared__ double red[kSumThreads];
    double d = 0.0;
    for (int k = threadIdx.x; k < n; k += kSumThreads) d += loss_part[k];
    red[threadIdx.x] = d;
    __syncthreads();
    for (int o = kSumThreads / 2; o >= 1; o >>= 1) {
      if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] / ((double)n * kNS);
    return;
  }
  const int i = blockIdx.x * kSumThreads + threadIdx.x;
  if (i >= kParams) return;
  const float* p = partial + i;
  float s = 0.0f, c = 0.0f, cc = 0.0f;
  constexpr int kRows = 25;  // loads at once
  for (int k0 = 0; k0 < parts; k0 += kRows) {
    float x[kRows];
#pragma unroll
    for (int k = 0; k < kRows; ++k) x[k] = k0 + k < parts ? p[(int64_t)(k0 + k) * kParams] : 0.0f;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      float e = 0.0f;
      two_sum_add(s, e, x[k]);
      two_sum_add(c, cc, e);
    }
  }
  float total = (float)((double)s + ((double)c + (double)cc));
  if (!(fabsf(total) < __int_as_float(0x7f800000))) {
    double d = 0.0;
    for (int k = 0; k < parts; ++k) d += (double)p[(int64_t)k * kParams];
    total = (float)d;
  }
  grad[i] = total;
}

}  // namespace
}  // namespace ws
}  // namespace cgb

using namespace cgb;
using namespace cgb::ws;

namespace {

// loss_part, loss: null, or the records' losses and where their mean goes; after: the
// kernel before it on the stream is the backward pass of the step.
int launch_wgrad(const void* d_feat, const void* d_hid, const void* d_dpre, const void* d_dout,
                 int n, float* d_partial, int n_parts, float* d_grad, const double* loss_part,
                 double* loss, bool after, cudaStream_t st) {
  if (n < 0 || n_parts < 1 || !d_feat || !d_hid || !d_dpre || !d_dout || !d_partial || !d_grad)
    return fail(CGB_ERR_ARG, "cgb_ws_wgrad_dev: bad arguments");
  int dev = 0, sms = 0;
  CGB_TRY_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
  CGB_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev),
               "cudaDeviceGetAttribute");
  // one CTA fits an SM: all of them at once, and no more slots than records; the rows left
  // over for the low parts of the slots with more than one record
  int parts = sms / kGroups < n_parts ? sms / kGroups : n_parts;
  if (parts > n) parts = n;
  if (parts < 1) parts = 1;
  int lows = n - parts < parts ? n - parts : parts;
  if (lows > n_parts - parts) lows = n_parts - parts;
  if (lows < 0) lows = 0;
  CGB_TRY_CUDA(cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kGradSmem),
               "cudaFuncSetAttribute(wgrad)");
  CGB_TRY_CUDA(launch_after(after, wgrad_kernel, kGroups * parts, kGradThreads, kGradSmem, st,
                            static_cast<const unsigned char*>(d_feat),
                            static_cast<const unsigned char*>(d_hid),
                            static_cast<const unsigned char*>(d_dpre),
                            static_cast<const unsigned char*>(d_dout), n, parts, lows, d_partial,
                            g_fault_skip_products),
               "wgrad_kernel launch");
  note_launch();
  CGB_TRY_CUDA(launch_after(true, reduce_kernel,
                            (kParams + kSumThreads - 1) / kSumThreads + (loss ? 1 : 0),
                            kSumThreads, 0, st, d_partial, parts + lows, d_grad, loss_part, n, loss),
               "reduce_kernel launch");
  note_launch();
  return CGB_OK;
}

}  // namespace

extern "C" int cgb_ws_wgrad_dev(const void* d_feat, const void* d_hid, const void* d_dpre,
                                const void* d_dout, int n, float* d_partial, int n_parts,
                                float* d_grad, void* stream) {
  return launch_wgrad(d_feat, d_hid, d_dpre, d_dout, n, d_partial, n_parts, d_grad, nullptr,
                      nullptr, false, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int cgb_ws_gradients_dev(const void* d_blob, const void* d_blobT, const void* d_feat,
                                    const float* d_target, int n, float s_out, void* d_hid,
                                    float* d_out, void* d_dout, void* d_dpre, double* d_loss_part,
                                    float* d_partial, int n_parts, double* d_loss, float* d_grad,
                                    void* stream) {
  if (!d_loss) return fail(CGB_ERR_ARG, "cgb_ws_gradients_dev: bad arguments");
  if (const int rc = forward_loss(d_blob, d_feat, n, d_hid, d_out, d_target, s_out, d_dout,
                                  d_loss_part, stream))
    return rc;
  if (const int rc = backward_after(d_blobT, d_dout, d_hid, n, d_dpre, stream)) return rc;
  return launch_wgrad(d_feat, d_hid, d_dpre, d_dout, n, d_partial, n_parts, d_grad, d_loss_part,
                      d_loss, n > 0, reinterpret_cast<cudaStream_t>(stream));
}
