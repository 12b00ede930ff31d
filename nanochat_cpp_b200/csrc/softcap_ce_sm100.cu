// Loss pass of the chunked lm_head under MX: per row of bf16 logits the log-sum-exp of the soft-capped logits
// (capped = softcap * tanh(z / softcap)) and the cross-entropy loss lse - capped[target]. Replaces nanochat-cpp's
// nanochat_softcap_ce_loss (src/nanochat/model/ops/softcap_ce_kernel.cu:62-116 with kGrad = false), same bits: the
// gradient is not written here, the quantizer's softcap-gradient prologue recomputes it from the logits and this
// kernel's lse and emits it as MX directly (quantize_sm100.cu).
// The fp32 sum of exponentials is order-sensitive, and lse feeds every gradient value, so the order is the
// reference's: 256 threads per row, thread t adds columns t * 8 + 2048 * i + k in order of i then k, a butterfly
// (xor 16..1) inside each warp, then the eight warp sums again by butterfly in warp 0. |capped| <= softcap, so
// exp(capped - softcap) needs no running maximum.
// A row of 32768 logits costs one tanh and one exp per element: the pass is bound by the SFU/ALU work, not by HBM
// (64 KB per row).
#include <algorithm>

#include <cuda_bf16.h>

#include "bf16x2_sm100.cuh"
#include "internal.h"

namespace mxb200 {

namespace {

constexpr int kThreads = 256;
constexpr int kVec = 8;

__device__ __forceinline__ float row_sum(float v, float* smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = static_cast<int>(threadIdx.x) & 31, warp = static_cast<int>(threadIdx.x) >> 5;
  if (lane == 0)
    smem[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < kThreads / 32 ? smem[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0)
      smem[0] = v;
  }
  __syncthreads();
  return smem[0];
}

__global__ void __launch_bounds__(kThreads) mxb200_softcap_ce_loss_kernel(const __nv_bfloat16* logits, int64_t ld,
                                                                          const int64_t* targets, int vocab, int padded,
                                                                          float softcap, float* loss, float* lse_out) {
  __shared__ float smem[kThreads / 32];
  const int64_t row = blockIdx.x;
  const __nv_bfloat16* z = logits + row * ld;
  const int64_t target = targets[row];
  if (target < 0) {  // ignored row: loss 0, lse left unset
    if (loss != nullptr && threadIdx.x == 0)
      loss[row] = 0.f;
    return;
  }
  float sum = 0.f;
  for (int j = static_cast<int>(threadIdx.x) * kVec; j < padded; j += kThreads * kVec) {
    const uint4 raw = *reinterpret_cast<const uint4*>(z + j);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int k = 0; k < kVec; ++k) {
      const float v = __uint_as_float((k & 1) ? (w[k >> 1] & 0xffff0000u) : (w[k >> 1] << 16));
      if (j + k < vocab)
        sum += expf(softcap * tanhf(v / softcap) - softcap);
    }
  }
  const float lse = softcap + logf(row_sum(sum, smem));
  if (threadIdx.x == 0) {
    if (loss != nullptr)
      loss[row] = lse - softcap * tanhf(__bfloat162float(z[target]) / softcap);
    if (lse_out != nullptr)
      lse_out[row] = lse;
  }
}

// ---- the small reductions around the chunks: one block each, a few microseconds for any batch of tokens

constexpr int kReduceThreads = 1024;

template <typename T>
__device__ __forceinline__ T block_sum(T v, T* smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = static_cast<int>(threadIdx.x) & 31, warp = static_cast<int>(threadIdx.x) >> 5;
  if (lane == 0)
    smem[warp] = v;
  __syncthreads();
  v = smem[lane];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(kReduceThreads) mxb200_count_valid_kernel(const int64_t* targets, int64_t n,
                                                                            int64_t* out) {
  __shared__ unsigned long long smem[kReduceThreads / 32];
  unsigned long long count = 0;
  for (int64_t i = threadIdx.x; i < n; i += kReduceThreads)
    count += targets[i] >= 0 ? 1u : 0u;
  count = block_sum(count, smem);
  if (threadIdx.x == 0)
    *out = static_cast<int64_t>(count);
}

// a thread's values in order, then the butterflies: the same sum on every run
__global__ void __launch_bounds__(kReduceThreads) mxb200_reduce_losses_kernel(const float* losses, int64_t n,
                                                                              const int64_t* num_valid, float* out) {
  __shared__ float smem[kReduceThreads / 32];
  float sum = 0.f;
  for (int64_t i = threadIdx.x; i < n; i += kReduceThreads)
    sum += losses[i];
  sum = block_sum(sum, smem);
  if (threadIdx.x == 0)
    *out = num_valid != nullptr ? sum / static_cast<float>(*num_valid) : sum;
}

// y = bf16(x * bf16(scale)), 16 bytes per thread and step; HBM-bound (4 bytes per value). torch's multiply by a 0-dim
// fp32 tensor converts that operand per element and took 95 us where this takes 17 on 16384 x 1536.
__global__ void __launch_bounds__(256) mxb200_scale_bf16_kernel(const uint4* x, const float* scale, uint4* y, int64_t n16) {
  const float f = __bfloat162float(__float2bfloat16(*scale));
  const uint32_t s2 = pack_bf16x2_rn(f, f);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < n16; i += static_cast<int64_t>(gridDim.x) * 256) {
    const uint4 v = x[i];
    y[i] = make_uint4(mul_bf16x2(v.x, s2), mul_bf16x2(v.y, s2), mul_bf16x2(v.z, s2), mul_bf16x2(v.w, s2));
  }
}

}  // namespace

}  // namespace mxb200

extern "C" int mxb200_softcap_ce_loss(const void* logits, int64_t rows, int64_t ld, const int64_t* targets, int vocab,
                                      int padded, float softcap, float* loss, float* lse, void* stream) {
  using namespace mxb200;
  DeviceInfo dev;
  if (int s = current_device(&dev); s != MXB200_OK)
    return s;
  if (logits == nullptr || targets == nullptr || (loss == nullptr && lse == nullptr))
    return MXB200_ERR_NULL;
  if (rows <= 0 || rows > 0x7fffffffLL || padded <= 0 || padded % kVec != 0 || ld < padded || ld % kVec != 0)
    return MXB200_ERR_SHAPE;
  if (vocab <= 0 || vocab > padded || !(softcap > 0.f))
    return MXB200_ERR_ARGUMENT;
  if (!aligned16(logits))
    return MXB200_ERR_ALIGNMENT;
  mxb200_softcap_ce_loss_kernel<<<static_cast<unsigned>(rows), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(logits), ld, targets, vocab, padded, softcap, loss, lse);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return launch_status();
}

extern "C" int mxb200_count_valid(const int64_t* targets, int64_t n, int64_t* out, void* stream) {
  using namespace mxb200;
  DeviceInfo dev;
  if (int s = current_device(&dev); s != MXB200_OK)
    return s;
  if (out == nullptr || (targets == nullptr && n > 0))
    return MXB200_ERR_NULL;
  if (n < 0)
    return MXB200_ERR_SHAPE;
  mxb200_count_valid_kernel<<<1, kReduceThreads, 0, static_cast<cudaStream_t>(stream)>>>(targets, n, out);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return launch_status();
}

extern "C" int mxb200_reduce_losses(const float* losses, int64_t n, const int64_t* num_valid, float* out, void* stream) {
  using namespace mxb200;
  DeviceInfo dev;
  if (int s = current_device(&dev); s != MXB200_OK)
    return s;
  if (out == nullptr || (losses == nullptr && n > 0))
    return MXB200_ERR_NULL;
  if (n < 0)
    return MXB200_ERR_SHAPE;
  mxb200_reduce_losses_kernel<<<1, kReduceThreads, 0, static_cast<cudaStream_t>(stream)>>>(losses, n, num_valid, out);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return launch_status();
}

extern "C" int mxb200_scale_bf16(const void* x, const float* scale, void* y, int64_t n, void* stream) {
  using namespace mxb200;
  DeviceInfo dev;
  if (int s = current_device(&dev); s != MXB200_OK)
    return s;
  if (x == nullptr || scale == nullptr || y == nullptr)
    return MXB200_ERR_NULL;
  if (n <= 0 || n % kVec != 0)
    return MXB200_ERR_SHAPE;
  if (!aligned16(x) || !aligned16(y))
    return MXB200_ERR_ALIGNMENT;
  const int64_t n16 = n / kVec;
  const int64_t blocks = std::min<int64_t>((n16 + 255) / 256, static_cast<int64_t>(dev.sms) * 8);
  mxb200_scale_bf16_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(x), scale, static_cast<uint4*>(y), n16);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return launch_status();
}
