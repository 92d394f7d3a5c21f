// Learned Jacobi warm start: training kernels and the standalone inference.
//
// The network and its feature vector are described in warmstart.cuh.  The
// training step is
//   prepare (once): features + exact pressure (FP64 tridiagonal solve) of
//                   logged step starts -> raw targets (p* - pe) / max|rt|
//   forward       : warmstart_conv.cu, hidden activations (BF16) kept for the
//                   backward pass
//   loss          : pred = s_out * o, MSE against the raw target; dL/do (BF16)
//   backward      : warmstart_conv.cu, the transposed convolutions with the
//                   ReLU masks -> pre-activation gradients (BF16)
//   weight grad   : warmstart_grad.cu
//   adam          : FP32 master parameters, then re-packed to BF16.
// The inference runs as in the BM kernel, a warp to a record (mma.sync m16n8k16
// BF16, FP32 accumulate); the training passes on tcgen05.
#include <cuda_runtime.h>

#include <cstdint>

#include "cgb_device.cuh"
#include "cgb_internal.h"
#include "warmstart.cuh"

namespace cgb {
namespace ws {

constexpr int kFeatBytes = kFeatRows * 16;

__device__ __forceinline__ uint16_t bf16_half(float f) { return (uint16_t)bf16_bits(f); }

// ---------------------------------------------------------------------------
// Packing: canonical FP32 -> BF16 blobs.
// ---------------------------------------------------------------------------
__global__ void pack_kernel(const float* __restrict__ prm, float s_out, float rm_scale,
                            unsigned char* __restrict__ blob, unsigned char* __restrict__ blobT) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = gridDim.x * blockDim.x;
  // W1 [6][64][8], tap 5 zero
  for (int i = tid; i < 6 * 64 * 8; i += nth) {
    const int tap = i / 512, co = (i / 8) % 64, ci = i % 8;
    const float w = tap < 5 ? prm[oW1 + (tap * 64 + co) * 8 + ci] : 0.0f;
    reinterpret_cast<uint16_t*>(blob + kOffW1)[i] = bf16_half(w);
  }
  // W2, W3 [5][64 out][64 in] as 64-channel rows (row = tap*64 + out)
  for (int i = tid; i < 2 * 5 * 64 * 64; i += nth) {
    const int l = i / (5 * 64 * 64), j = i % (5 * 64 * 64);
    const int row = j / 64, ci = j % 64;
    const float w = prm[(l ? oW3 : oW2) + j];
    *reinterpret_cast<uint16_t*>(blob + (l ? kOffW3 : kOffW2) + swz64(row, ci >> 3) +
                                 (ci & 7) * 2) = bf16_half(w);
  }
  // W4 [5][8 out][64 in]; outputs 1..7 zero
  for (int i = tid; i < 5 * 8 * 64; i += nth) {
    const int row = i / 64, ci = i % 64, tap = row / 8, co = row % 8;
    const float w = co == 0 ? prm[oW4 + tap * 64 + ci] : 0.0f;
    *reinterpret_cast<uint16_t*>(blob + kOffW4 + swz64(row, ci >> 3) + (ci & 7) * 2) =
        bf16_half(w);
  }
  float* bias = reinterpret_cast<float*>(blob + kOffBias);
  for (int i = tid; i < kBiasFloats; i += nth) {
    float b = 0.0f;
    if (i < 64) b = prm[ob1 + i];
    else if (i < 128) b = prm[ob2 + i - 64];
    else if (i < 192) b = prm[ob3 + i - 128];
    else if (i == 192) b = prm[ob4];
    else if (i == 200) b = s_out;
    else if (i == 201) b = rm_scale;
    bias[i] = b;
  }
  if (!blobT) return;
  // W4T [6 taps][64 out(=in of W4)][8 in(=out of W4)]: W4T[t][ci][co] = W4[4-t][co][ci]
  for (int i = tid; i < 6 * 64 * 8; i += nth) {
    const int tap = i / 512, ci = (i / 8) % 64, co = i % 8;
    const float w = (tap < 5 && co == 0) ? prm[oW4 + (4 - tap) * 64 + ci] : 0.0f;
    reinterpret_cast<uint16_t*>(blobT + kOffT4)[i] = bf16_half(w);
  }
  // W3T, W2T [5][64][64]: WT[t][ci][co] = W[4-t][co][ci]
  for (int i = tid; i < 2 * 5 * 64 * 64; i += nth) {
    const int l = i / (5 * 64 * 64), j = i % (5 * 64 * 64);
    const int tap = j / 4096, ci = (j / 64) % 64, co = j % 64;
    const float w = prm[(l ? oW2 : oW3) + ((4 - tap) * 64 + co) * 64 + ci];
    const int row = tap * 64 + ci;
    *reinterpret_cast<uint16_t*>(blobT + (l ? kOffT2 : kOffT3) + swz64(row, co >> 3) +
                                 (co & 7) * 2) = bf16_half(w);
  }
}

// ---------------------------------------------------------------------------
// Prepare: features, extrapolated guess, max|rt| and the raw target of each
// logged record (one warp per record).  Record: [6][256] = Y/m, p1, p2, v,
// x, {rho, ...}.  The exact pressure solves p_s + (1/m_s)(l_s p_{s-1} +
// p_{s+1}) = Y_s/m_s (the system the Jacobi sweep iterates) in FP64.
// ---------------------------------------------------------------------------
__global__ void prepare_kernel(const float* __restrict__ rec, int n, const float* __restrict__ rm_g,
                               float rm_scale, unsigned char* __restrict__ feat,
                               float* __restrict__ target, float* __restrict__ nr_out,
                               double* __restrict__ work) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (wid >= n) return;
  const float* r = rec + (int64_t)wid * 6 * 256;
  const int base = lane * 8;
  float Yrm[8], p1[8], p2[8], v[8], x[8], rm[8], pe[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    Yrm[k] = r[0 * 256 + base + k];
    p1[k] = r[1 * 256 + base + k];
    p2[k] = r[2 * 256 + base + k];
    v[k] = r[3 * 256 + base + k];
    x[k] = r[4 * 256 + base + k];
    rm[k] = rm_g[base + k];
  }
  const float rho = r[5 * 256];
  unsigned char* f = feat + (int64_t)wid * kFeatBytes;
  // rows outside the unit are zero
  for (int i = lane; i < 8; i += 32) {
    reinterpret_cast<uint4*>(f)[i] = make_uint4(0, 0, 0, 0);
  }
  for (int i = lane; i < kFeatRows - 264; i += 32)
    reinterpret_cast<uint4*>(f)[264 + i] = make_uint4(0, 0, 0, 0);
  const float nr = make_features(Yrm, p1, p2, v, x, rm, rho, rm_scale, pe, f, 8, lane);
  // exact solve (lane 0, FP64 Thomas); work: [n][2][256]
  double* c = work + (int64_t)wid * 512;
  double* y = c + 256;
  if (lane == 0) {
    // row s: lower a_s = rm_s * l_s (s >= 1), diag 1, upper b_s = rm_s
    double cp = 0.0, yp = 0.0;
    for (int s = 0; s < 256; ++s) {
      const double rs = (double)rm_g[s];
      const double a = (s >= 1 && s < 254) ? rs : 0.0;
      const double b = s < 255 ? rs : 0.0;
      const double den = 1.0 - a * cp;
      cp = b / den;
      yp = ((double)r[s] - a * yp) / den;
      c[s] = cp;
      y[s] = yp;
    }
    for (int s = 254; s >= 0; --s) y[s] -= c[s] * y[s + 1];
  }
  __syncwarp();
  const float inr = nr > 0.0f ? 1.0f / nr : 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    target[(int64_t)wid * 256 + base + k] = (float)((y[base + k] - (double)pe[k]) * (double)inr);
  if (lane == 0) nr_out[wid] = nr;
}

__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes, int tid, int nth) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  uint4* d = reinterpret_cast<uint4*>(dst);
  for (int i = tid; i < bytes / 16; i += nth) d[i] = s[i];
}

// ---------------------------------------------------------------------------
// Loss: pred = s_out * o; L = sum (pred - target)^2 / (n * 256);
// dL/do -> channel 0 of 8-channel rows (BF16), channels 1..7 zero.
// ---------------------------------------------------------------------------
__global__ void loss_kernel(const float* __restrict__ out, const float* __restrict__ target, int n,
                            float s_out, unsigned char* __restrict__ dout,
                            double* __restrict__ loss_part) {
  __shared__ double red[256];
  const int rec = blockIdx.x, s = threadIdx.x;
  const float e = s_out * out[(int64_t)rec * 256 + s] - target[(int64_t)rec * 256 + s];
  const float gsc = 2.0f * s_out / ((float)n * 256.0f);
  uint4 w = make_uint4(bf16_bits(gsc * e), 0, 0, 0);
  reinterpret_cast<uint4*>(dout + (int64_t)rec * 256 * 16)[s] = w;
  red[s] = (double)e * (double)e;
  __syncthreads();
  for (int o = 128; o >= 1; o >>= 1) {
    if (s < o) red[s] += red[s + o];
    __syncthreads();
  }
  if (s == 0) loss_part[rec] = red[0];
}

__global__ void adam_kernel(float* __restrict__ prm, const float* __restrict__ grad,
                            float* __restrict__ m, float* __restrict__ v, float lr, float b1,
                            float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  const float g = grad[i];
  const float mi = b1 * m[i] + (1.0f - b1) * g;
  const float vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  prm[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// Standalone inference through the BM kernel's fused routine: one warp per
// record, 4 warps per CTA sharing the weights.
constexpr int kInferSmem = kBlobBytes + 4 * kWarpScratch;

__global__ void __launch_bounds__(128) infer_kernel(const unsigned char* __restrict__ blob,
                                                    const unsigned char* __restrict__ feat, int n,
                                                    float* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  copy16(sm, blob, kBlobBytes, tid, 128);
  unsigned char* scratch = sm + kBlobBytes + warp * kWarpScratch;
  for (int i = lane; i < kWarpScratch / 16; i += 32)
    reinterpret_cast<uint4*>(scratch)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int rec = blockIdx.x * 4 + warp; rec < n; rec += gridDim.x * 4) {
    const uint4* f = reinterpret_cast<const uint4*>(feat + (int64_t)rec * kFeatBytes);
    for (int i = lane; i < 256; i += 32) reinterpret_cast<uint4*>(scratch)[8 + i] = f[8 + i];
    __syncwarp();
    infer_unit(sm, scratch, lane);
    const float* o = reinterpret_cast<const float*>(scratch + kOffOut);
    for (int i = lane; i < 256; i += 32) out[(int64_t)rec * 256 + i] = o[i];
    __syncwarp();
  }
}

int grid_for(int n, int per) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long want = ((long long)n + per - 1) / per;
  long long cap = (long long)sms * 4;
  return (int)(want < cap ? (want < 1 ? 1 : want) : cap);
}

template <typename K>
int set_smem(K kernel, int bytes, const char* what) {
  CGB_TRY_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes),
               what);
  return CGB_OK;
}

}  // namespace ws
}  // namespace cgb

using namespace cgb;
using namespace cgb::ws;

extern "C" int cgb_ws_blob_bytes(void) { return kBlobBytes; }
extern "C" int cgb_ws_blobT_bytes(void) { return kBlobTBytes; }
extern "C" int cgb_ws_param_count(void) { return kParams; }

extern "C" int cgb_ws_pack_dev(const float* d_params, float s_out, float rm_scale, void* d_blob,
                               void* d_blobT, void* stream) {
  if (!d_params || !d_blob) return fail(CGB_ERR_ARG, "cgb_ws_pack_dev: null pointer");
  if ((reinterpret_cast<uintptr_t>(d_blob) & 15) || (reinterpret_cast<uintptr_t>(d_blobT) & 15))
    return fail(CGB_ERR_ARG, "cgb_ws_pack_dev: blobs must be 16-byte aligned");
  pack_kernel<<<64, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      d_params, s_out, rm_scale, static_cast<unsigned char*>(d_blob),
      static_cast<unsigned char*>(d_blobT));
  CGB_TRY_CUDA(cudaGetLastError(), "pack_kernel launch");
  note_launch();
  return CGB_OK;
}

extern "C" int cgb_ws_prepare_dev(const float* d_rec, int n, const float* d_rm, float rm_scale,
                                  void* d_feat, float* d_target, float* d_nr, double* d_work,
                                  void* stream) {
  if (n == 0) return CGB_OK;
  if (n < 0 || !d_rec || !d_rm || !d_feat || !d_target || !d_nr || !d_work)
    return fail(CGB_ERR_ARG, "cgb_ws_prepare_dev: bad arguments");
  const int warps = 8;
  prepare_kernel<<<(n + warps - 1) / warps, warps * 32, 0,
                   reinterpret_cast<cudaStream_t>(stream)>>>(
      d_rec, n, d_rm, rm_scale, static_cast<unsigned char*>(d_feat), d_target, d_nr, d_work);
  CGB_TRY_CUDA(cudaGetLastError(), "prepare_kernel launch");
  note_launch();
  return CGB_OK;
}

extern "C" int cgb_ws_loss_dev(const float* d_out, const float* d_target, int n, float s_out,
                               void* d_dout, double* d_loss_part, void* stream) {
  if (n == 0) return CGB_OK;
  if (n < 0 || !d_out || !d_target || !d_dout || !d_loss_part)
    return fail(CGB_ERR_ARG, "cgb_ws_loss_dev: bad arguments");
  loss_kernel<<<n, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      d_out, d_target, n, s_out, static_cast<unsigned char*>(d_dout), d_loss_part);
  CGB_TRY_CUDA(cudaGetLastError(), "loss_kernel launch");
  note_launch();
  return CGB_OK;
}

extern "C" int cgb_ws_adam_dev(float* d_params, const float* d_grad, float* d_m, float* d_v,
                               int step, float lr, float beta1, float beta2, float eps,
                               void* stream) {
  if (!d_params || !d_grad || !d_m || !d_v || step < 1)
    return fail(CGB_ERR_ARG, "cgb_ws_adam_dev: bad arguments");
  const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
  adam_kernel<<<(kParams + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      d_params, d_grad, d_m, d_v, lr, beta1, beta2, eps, c1, c2);
  CGB_TRY_CUDA(cudaGetLastError(), "adam_kernel launch");
  note_launch();
  return CGB_OK;
}

extern "C" int cgb_ws_infer_dev(const void* d_blob, const void* d_feat, int n, float* d_out,
                                void* stream) {
  if (n == 0) return CGB_OK;
  if (n < 0 || !d_blob || !d_feat || !d_out)
    return fail(CGB_ERR_ARG, "cgb_ws_infer_dev: bad arguments");
  if (set_smem(infer_kernel, kInferSmem, "cudaFuncSetAttribute(infer)")) return CGB_ERR_CUDA;
  infer_kernel<<<grid_for(n, 4), 128, kInferSmem, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const unsigned char*>(d_blob), static_cast<const unsigned char*>(d_feat), n,
      d_out);
  CGB_TRY_CUDA(cudaGetLastError(), "infer_kernel launch");
  note_launch();
  return CGB_OK;
}
