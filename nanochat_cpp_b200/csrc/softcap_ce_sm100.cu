// Loss pass of the chunked lm_head under MX: per row of bf16 logits the log-sum-exp of the soft-capped logits
// (capped = softcap * tanh(z / softcap)) and the cross-entropy loss lse - capped[target]. Replaces nanochat-cpp's
// nanochat_softcap_ce_loss (src/nanochat/model/ops/softcap_ce_kernel.cu:62-116 with kGrad = false), same bits: the
// gradient is not written here, the quantizer's softcap-gradient prologue recomputes it from the logits and this
// kernel's lse and emits it as MX directly (quantize_sm100.cu).
// The fp32 sum of exponentials is order-sensitive, and lse feeds every gradient value, so the order is the
// reference's: 256 threads per row, thread t adds columns t * 8 + 2048 * i + k in order of i then k, a butterfly
// (xor 16..1) inside each warp, then the eight warp sums again by butterfly in warp 0. |capped| <= softcap, so
// exp(capped - softcap) needs no running maximum.
#include <algorithm>

#include <cuda_bf16.h>

#include "bf16x2_sm100.cuh"
#include "internal.h"
#include "ptx_sm100.cuh"
#include "softcap_table_sm100.cuh"

namespace mxb200 {

namespace {

constexpr int kThreads = 256;
constexpr int kVec = 8;

// The row's sum over its 256 threads in the reference's order. `bar`: the group's named barrier; smem: 8 floats per group.
__device__ __forceinline__ float row_sum(float v, float* smem, int bar) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = static_cast<int>(threadIdx.x) & 31, warp = (static_cast<int>(threadIdx.x) >> 5) & 7;
  if (lane == 0)
    smem[warp] = v;
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(kThreads) : "memory");
  v = lane < kThreads / 32 ? smem[lane] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(kThreads) : "memory");  // before the next row's sums overwrite these
  return v;
}

struct LossParams {
  const __nv_bfloat16* logits;
  int64_t ld;
  const int64_t* targets;
  int64_t rows;
  int vocab, padded;
  float softcap;
  float* loss;
  float* lse;
};

// Adds the terms of eight logits, the first `left` of them inside the vocabulary.
__device__ __forceinline__ float add_direct(float sum, uint4 z, int left, float at_zero, float softcap) {
  const uint32_t w[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
  for (int k = 0; k < kVec; ++k) {
    const float v = (k & 1) ? hi_f32(w[k >> 1]) : lo_f32(w[k >> 1]);
    if (k < left)
      sum += v == 0.f ? at_zero : softcap_loss_term(v, softcap);
  }
  return sum;
}

// The same beside the table's path, where it is rare: out of the loop's registers and instructions.
__device__ __noinline__ float add_direct_outlined(float sum, uint4 z, int left, float at_zero, float softcap) {
  return add_direct(sum, z, left, at_zero, softcap);
}

// The table of exp(capped - softcap) (softcap_table_sm100.cuh says why) of this kernel covers |z| in [2^-25, 2^7), 4096
// magnitudes, so that one packed subtraction and an or per two logits tell whether a lookup is allowed. Entries of positive
// logits sit at the front of shared memory and those of negative ones 128 KB further on: the address is the logit's 16
// bits times 4, a shift and a mask. That takes 144 KB, too much for two CTAs per SM, so one with four groups of threads serves it.
constexpr uint32_t kTermLow = (127 - 25) << 7;
constexpr uint32_t kTermMagnitudes = 4096;
constexpr uint32_t kLossTableBytes = 0x8000 * 4 + kTermMagnitudes * 4;
static_assert(kTermLow + kTermMagnitudes == kLogitHigh && kLossTableBytes <= 232448);

// A row per 256 threads, kGroups rows at a time per CTA, persistent over rows. With the table it is bound by shared
// memory: 32 random reads per instruction take about 3.6 bank cycles, so 2048 x 32768 logits need 27 us of them at 1.85
// GHz against 20 us for the bytes; it takes 41.5 us (the path to shared memory 71% busy); evaluated directly they took 106 us.
template <bool kTable, int kGroups, int kCtas>
__global__ void __launch_bounds__(kThreads * kGroups, kCtas) mxb200_softcap_ce_loss_kernel(const LossParams p) {
  extern __shared__ __align__(16) float table[];
  __shared__ float smem[kGroups][kThreads / 32];
  const int group = static_cast<int>(threadIdx.x) / kThreads, t = static_cast<int>(threadIdx.x) % kThreads;
  // rows go round the CTAs first and their groups second, so that every SM gets the same number of rows
  const int64_t first_row = blockIdx.x + static_cast<int64_t>(group) * gridDim.x;
  const int64_t row_step = static_cast<int64_t>(gridDim.x) * kGroups;
  constexpr int kStep = kThreads * kVec;
  // vectors in flight ahead of the one being added up (the additions are a serial chain per thread); those of a row's
  // start are asked for before the row ahead of it is summed up. The table is made while the kernel before ends.
  constexpr int kAhead = kTable ? 4 : 2;
  uint4 next[kAhead];
  const auto load = [&](int64_t row, int j) {
    return row < p.rows && j < p.padded ? *reinterpret_cast<const uint4*>(p.logits + row * p.ld + j)
                                        : make_uint4(0u, 0u, 0u, 0u);
  };
  if constexpr (kTable) {
    for (uint32_t i = threadIdx.x; i < kTermMagnitudes; i += kThreads * kGroups) {
      const float th = softcap_tanh(__uint_as_float((kTermLow + i) << 16), p.softcap);  // of -z: -th
      table[i] = expf(p.softcap * th - p.softcap);
      table[0x8000 + i] = expf(p.softcap * -th - p.softcap);
    }
    __syncthreads();
  }
  grid_dependency_wait();
#pragma unroll
  for (int k = 0; k < kAhead; ++k)
    next[k] = load(first_row, t * kVec + k * kStep);
  const float at_zero = softcap_loss_term(0.f, p.softcap);
  const uint32_t table_base = static_cast<uint32_t>(__cvta_generic_to_shared(table)) - 4 * kTermLow;
  for (int64_t row = first_row; row < p.rows; row += row_step) {
    const int64_t target = p.targets[row];
    float sum = 0.f;
    const auto add = [&](const uint4& raw, int j) {
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
      // no bit above the 12 of a table index may be set in any (magnitude - low); a borrow out of the low half sets its
      // own upper bits
      uint32_t outside = 0u;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        outside |= (w[k] & 0x7fff7fffu) - kTermLow * 0x10001u;
      if (kTable && j + kVec <= p.vocab && (outside & 0xf000f000u) == 0u) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sum += load_shared_f32(table_base + ((w[k] << 2) & 0x3fffcu));
          sum += load_shared_f32(table_base + ((w[k] >> 14) & 0x3fffcu));
        }
      } else {
        sum = kTable ? add_direct_outlined(sum, raw, p.vocab - j, at_zero, p.softcap)
                     : add_direct(sum, raw, p.vocab - j, at_zero, p.softcap);
      }
    };
    if (target >= 0) {
      for (int j = t * kVec; j < p.padded; j += kAhead * kStep) {
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          const int at = j + k * kStep;
          const uint4 raw = next[k];
          next[k] = load(row, at + kAhead * kStep);
          if (at < p.padded)
            add(raw, at);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      next[k] = load(row + row_step, t * kVec + k * kStep);
    if (target < 0) {  // ignored row: loss 0, lse left unset
      if (p.loss != nullptr && t == 0)
        p.loss[row] = 0.f;
      continue;
    }
    const float lse = p.softcap + logf(row_sum(sum, smem[group], 1 + group));
    if (t == 0) {
      if (p.loss != nullptr)
        p.loss[row] = lse - p.softcap * tanhf(__bfloat162float(p.logits[row * p.ld + target]) / p.softcap);
      if (p.lse != nullptr)
        p.lse[row] = lse;
    }
  }
}

template <bool kTable, int kGroups, int kCtas>
int launch_loss(const LossParams& p, const DeviceInfo& dev, cudaStream_t stream) {
  constexpr auto kernel = mxb200_softcap_ce_loss_kernel<kTable, kGroups, kCtas>;
  constexpr size_t smem = kTable ? kLossTableBytes : 0;
  static std::atomic<int> configured_for{-1};
  if (kTable && configured_for.load() != dev.device) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess)
      return MXB200_ERR_LAUNCH;
    configured_for.store(dev.device);
  }
  const int64_t ctas = std::min<int64_t>(p.rows, static_cast<int64_t>(dev.sms) * kCtas);
  return launch_kernel(kernel, static_cast<unsigned>(ctas), kThreads * kGroups, smem, stream, p);
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
  grid_dependency_wait();
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
  grid_dependency_wait();
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
  grid_dependency_wait();
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
  const LossParams p{static_cast<const __nv_bfloat16*>(logits), ld, targets, rows, vocab, padded, softcap, loss, lse};
  auto* s = static_cast<cudaStream_t>(stream);
  // the table is worth making where a CTA looks up at least three times its entries (a CTA makes 8 per thread)
  if (rows * padded >= 3 * 2 * static_cast<int64_t>(kTermMagnitudes) * std::min<int64_t>(rows, dev.sms))
    return launch_loss<true, 4, 1>(p, dev, s);
  return launch_loss<false, 1, 6>(p, dev, s);
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
  return launch_kernel(mxb200_count_valid_kernel, 1, kReduceThreads, 0, static_cast<cudaStream_t>(stream), targets, n, out);
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
  return launch_kernel(mxb200_reduce_losses_kernel, 1, kReduceThreads, 0, static_cast<cudaStream_t>(stream), losses, n,
                       num_valid, out);
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
  return launch_kernel(mxb200_scale_bf16_kernel, static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream),
                       static_cast<const uint4*>(x), scale, static_cast<uint4*>(y), n16);
}
