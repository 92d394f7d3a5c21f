// What the BM/OHC kernels (bm_step.cu: a warp per unit, bm_quad.cu: four warps
// per unit) share: their arguments and the reference-arithmetic helpers.
#pragma once

#include <cuda_runtime.h>

#include "cgb_device.cuh"
#include "cochlea_gb300.h"

namespace cgb {

struct BMArgs {
  const float* secp;   // [8][256]: 1/M, 1/m, R, S, Q, S_ohc, S_tm, R_tm
  const float* gamma;  // [P][256]
  const cgb_unit* units;
  int n_units;
  const float* in;
  float* out;
  // host mirror of out (pinned, mapped): its byte offset from out, or 0 for
  // none; a row's host address is its device address plus the offset
  long long host_delta;
  int32_t* failed;
  float* conv;  // [rows][3] mean dt, substeps, mean outer iterations per sample
  cgb_unit_stats* stats;
  int32_t* work;
  float ratio, nas, al, e1, e2, nw, ar, dx2, dxa0, na1, na2, gme, sow;
  float dt0, dtmin, dtmax;
  // the reference's float constants 1/Ts, 1/sigma_ow (each formed in double
  // and rounded, src/cochlea.cu:1099,1105) and time_step_out
  float fs_f, rsow, tout_f;
  // sigma_ow is a power of two (its reciprocal rsow is exact), so x / sigma_ow
  // is x * rsow bit for bit
  int ow_pow2;
  int jfast, jslow, max_outer, max_sub;
  // tolerance mode (jacobi_mode 2)
  float jtol;
  int jcap, guess, learn_every;
  const unsigned char* ws_blob;  // packed network weights (guess 2)
  float* log;                    // training records [6][256] (optional)
  long long log_cap;
  int log_every;
  int* log_count;
};

// CUDA's tanhf and __fdividef on a pair (ARITH 1).
__device__ __forceinline__ float2 tanhf2(float2 x) { return f2(tanhf(x.x), tanhf(x.y)); }
__device__ __forceinline__ float2 fdividef2(float2 a, float2 b) {
  return f2(__fdividef(a.x, b.x), __fdividef(a.y, b.y));
}

// Sweeps of the reference schedule: of the first two iterations of a step, and of
// the others.  Both kernels have instances that know these counts.
constexpr int kSlowSweeps = 20, kFastSweeps = 2;

// Launches the four-warps-per-unit kernel (fixed sweep counts); the status.
int bm_quad_launch(const BMArgs& A, int controller, int arith, cudaStream_t st);
// Most Jacobi sweeps of one solve that the four-warp kernel's halo carries.
constexpr int kQuadMaxSweeps = 32;

}  // namespace cgb
