// The AC filter as a matrix product on the 5th-generation tensor cores, exact
// to the last bit that matters: the pieces of ihc_tensor.cu's kernel.
//
// A tile is 128 output rows x 64 sections.  Its filter outputs are T x, T the
// 128 x 384 band of the taps and x the 384 rows that end with the tile.  Both
// factors are written as fixed-point numbers in base 2^9, of six and five digits,
//   x = 2^(e-8)  sum_i X_i 2^(-9 i),   b = 2^(eb-8) sum_j B_j 2^(-9 j),
// |X_i|, |B_j| <= 256 (rounded to nearest, so signed), e and eb the exponents
// of the largest magnitude of a section's 384 rows and of the taps.  Integers
// up to 256 are exact in BF16.  The 20 digit pairs with i + j <= 5 go to six
// accumulators G_m, m = i + j:
//   T x = 2^(e+eb-16) sum_m G_m 2^(-9 m)  +  the digits' remainders (at most 2^(e-54)
// of a value of x, 2^(eb-45) of a tap) and the pairs left out (about 2^-50 of the
// product of the scales; 2^-41 with the 15 pairs up to i + j = 4).
// An FP32 accumulator holds exact integers while no partial sum reaches 2^24.  A
// partial sum of G_m is at most M_m = 256 (S_0 + .. + S_m), S_j the sum of |B_j| over
// the taps.  The filter is taken only if that holds G_0 and G_1 (0.61 x 2^24 for the
// default one); G_2 to G_4 (1.11, 1.46, 1.46) are told to be exact from their final values:
// if a partial sum had reached 2^24, what is left of M_m could not bring the sum back
// below 2^25 - M_m.  What G_5 may have lost counts as an error of the sum (bounds:
// ihc_tensor_taps).
//
// T has one value per diagonal.  With the rows of x stored in reverse order its
// band is a Hankel matrix (element (r, k') depends on r + k'), and a Hankel
// matrix of 8 x 8 core matrices needs only one core matrix per block diagonal:
// the row and the column stride of the shared-memory descriptor are the same
// 128 bytes, and a digit of the whole 128 x 384 matrix takes 63 core matrices
// (8 KB) instead of 96 KB.
//
// The instruction reads both operands from shared memory at 128 bytes a cycle:
// 128 x N x 16 takes 32 + N / 4 cycles up to N = 128 (measured 40.8 at N = 32,
// 48.8 at N = 64), so a tile of 64 sections costs 20% more than one of 32.
// Twice that again if one thread issues it in a divergent branch (55 to 82
// cycles): the issuing warp stays converged and an elected lane's predicate
// guards the instruction.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace cgb {
namespace tfir {

constexpr int kRows = 128;           // output rows of a tile (M)
constexpr int kCols = 64;            // sections of a tile (N)
constexpr int kDepth = 384;          // rows of x of a tile (K)
constexpr int kHalf = kDepth / 2;    // rows in one of the two buffers of a digit
constexpr int kDigits = 5;           // of a tap
constexpr int kRowDigits = 6;        // of a value of x
constexpr int kSums = 6;             // accumulators
constexpr int kMaxTaps = kDepth - kRows + 1;
constexpr int kCores = (kRows + kDepth) / 8 - 1;  // block diagonals of the band
constexpr int kTapDigit = kCores * 128;           // bytes of a digit of the band
constexpr int kTapBytes = kDigits * kTapDigit;
constexpr int kBlockBytes = kCols * 16;           // eight rows of a digit of x
constexpr int kHalfBytes = kHalf / 8 * kBlockBytes;
constexpr uint32_t kTmemCols = 512;               // six accumulators of 64 columns

__device__ __forceinline__ uint32_t saddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The next digit of a remainder r (in units of the last digit, |r| <= 0.5, or
// the whole scaled value for the first): y = 512 r (or r) = digit + remainder.
__device__ __forceinline__ float digit(float& r, float up) {
  const float magic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
  const float t = __fmaf_rn(r, up, magic);
  const float d = __fsub_rn(t, magic);
  r = __fmaf_rn(r, up, -d);
  return d;
}

// Two BF16 digits (exact: small integers) in one register, the first in the
// low half.
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}

// Shared-memory operand descriptor without swizzle: start address, distance of
// the core matrices that follow each other in K (leading) and in M or N
// (stride), in bytes.
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t k_bytes, uint32_t mn_bytes) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(k_bytes >> 4) << 16) |
         ((uint64_t)(mn_bytes >> 4) << 32) | (1ull << 46);
}

// kind::f16 instruction: FP32 accumulators, BF16 operands, both K-major,
// 128 x 64.
constexpr uint32_t kInstr = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kCols / 8) << 17) |
                            ((uint32_t)(kRows / 16) << 24);

// One lane of the warp (all lanes call): the one whose predicate issues.
__device__ __forceinline__ uint32_t elected() {
  uint32_t e;
  asm volatile("{ .reg .pred q; elect.sync _|q, 0xffffffff; selp.u32 %0, 1, 0, q; }" : "=r"(e));
  return e;
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate,
                                    uint32_t issue, uint32_t instr = kInstr) {
  asm volatile(
      "{ .reg .pred p, q; setp.ne.b32 p, %4, 0; setp.ne.b32 q, %5, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d),
      "l"(a), "l"(b), "r"(instr), "r"(accumulate), "r"(issue)
      : "memory");
}

// The products of one digit i of x, half h of its rows, with the tap digits j
// up to 5 - i; called by a converged warp.  Accumulator m at column 64 m of
// tmem, started by its first product of the tile.
__device__ __forceinline__ void products(uint32_t taps, uint32_t rows, uint32_t tmem, int i,
                                         int h, uint32_t issue) {
  const uint64_t b0 = operand(rows, kBlockBytes, 128);
  const uint64_t a0 = operand(taps + h * (kHalf / 8) * 128, 128, 128);
#pragma unroll 1
  for (int j = 0; j < kDigits && j + i < kSums; ++j) {
    const uint32_t add = h > 0 || (i > 0 && i + j < kDigits) || i > 1 ? 1u : 0u;
    const uint64_t a = a0 + (uint64_t)((j * kTapDigit) >> 4);
    const uint32_t d = tmem + kCols * (i + j);
#pragma unroll
    for (int k = 0; k < kHalf / 16; ++k)
      mma(d, a + ((k * 256) >> 4), b0 + ((k * 2 * kBlockBytes) >> 4), k > 0 ? 1u : add, issue);
  }
}

__device__ __forceinline__ void commit(uint64_t* mbar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          saddr(mbar))
      : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {  // one whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   saddr(slot)),
               "r"(kTmemCols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_free(uint32_t tmem) {  // the same warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
               "r"(kTmemCols));
}

// Eight consecutive columns of this lane's accumulator row.
__device__ __forceinline__ void tmem_load8(uint32_t addr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(addr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// Four, and back.
__device__ __forceinline__ void tmem_load4(uint32_t addr, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_store4(uint32_t addr, const float (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
               "r"(__float_as_uint(v[3]))
               : "memory");
}
__device__ __forceinline__ void tmem_wait_stores() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_loads() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

}  // namespace tfir
}  // namespace cgb
