// Host side of the IHC / lambda kernel with the AC filter on the tensor cores.
#pragma once

#include <cuda_runtime.h>

#include "ihc_common.cuh"

namespace cgb {

// Shorter filters stay on the FP32 pipe: a tile costs about the same for any length (and
// frames of few rows, tensor_faster of ihc_lambda.cu).
// JND sweep, FP32 against tensor cores: 32 taps 13.3 / 17.0 ms, 48 16.2 / 17.0, 64
// 19.2 / 17.1, 128 31.2 / 18.1; 286,000 rows: 48 taps 1.93 / 1.94, 64 2.28 / 1.98.
constexpr int kTensorMinTaps = 64;
constexpr int kTensorTileRows = 128;
constexpr int kTensorSections = 64;

// Whether the filters' lengths fit the kernel (taps of one tile, shared memory).
bool ihc_tensor_fits(int n_ac, int n_dc);
// What the kernel takes from the AC taps (scaled, as they are uploaded).
struct TensorTaps {
  int exp_b;    // 2^(exp_b-1) <= largest |tap| < 2^exp_b
  float floor;  // largest error of a sum, in units of the accumulators (head of ihc_tensor.cu)
  float limit;  // of the third to fifth accumulator: exact below
};
// False: taps whose digit products the accumulators do not hold.
bool ihc_tensor_taps(const float* taps, int n_ac, float scale, TensorTaps* out);
int ihc_tensor_launch(const IHCArgs& A, const float* d_v, int n_runs, const TensorTaps& taps,
                      cudaStream_t st);

}  // namespace cgb
