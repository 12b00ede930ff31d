// Tables over bf16 logits for the softcap kernels. Device-only.
//
// tanh(z / softcap), and for the loss pass exp(softcap * tanh(z / softcap) - softcap), are functions of one bf16 value:
// 65536 inputs at most, of which a chunk of logits meets a few thousand some 67 million times. A CTA therefore evaluates
// them once per |z| below 2^7, from 2^-16 on for the gradient's tanh and from 2^-25 on for the loss's terms, into shared memory
// and then looks them up, with the bits of the direct evaluation because the entries are made by it. A division, a tanhf and
// an expf are about 60 instructions; a lookup is 3 plus a shared-memory read whose 32 random addresses take about 3.5 bank
// cycles. Values outside the range are evaluated directly.
#pragma once

#include <cstdint>

#include <cuda_bf16.h>

namespace mxb200 {

constexpr uint32_t kLogitLow = (127 - 16) << 7;  // bf16 bits of 2^-16
constexpr uint32_t kLogitHigh = (127 + 7) << 7;  // bf16 bits of 2^7, exclusive
constexpr uint32_t kLogitEntries = kLogitHigh - kLogitLow;  // magnitudes

// The reference's expressions (src/nanochat/model/ops/softcap_ce_kernel.cu:49-54, 75-80).
__device__ __forceinline__ float softcap_tanh(float z, float softcap) {
  return tanhf(z / softcap);
}

__device__ __forceinline__ float softcap_loss_term(float z, float softcap) {
  return expf(softcap * tanhf(z / softcap) - softcap);
}

__device__ __forceinline__ float load_shared_f32(uint32_t address) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(address));
  return v;
}

// tanh(z / softcap) of the low (half 0) or high 16 bits of w. The table holds tanh of the magnitudes from kLogitLow on (tanhf
// is odd); m: w without the signs.
__device__ __forceinline__ float logit_tanh(const float* table, uint32_t w, uint32_t m, int half) {
  const float magnitude = table[static_cast<int>(half ? m >> 16 : m & 0xffffu) - static_cast<int>(kLogitLow)];
  const uint32_t sign = (half ? w : w << 16) & 0x80000000u;
  return __uint_as_float(__float_as_uint(magnitude) ^ sign);
}

// Whether every magnitude in 4 packed words has an entry.
__device__ __forceinline__ bool magnitudes_in_table(const uint32_t (&m)[4]) {
  uint32_t lo = m[0], hi = m[0];
#pragma unroll
  for (int k = 1; k < 4; ++k) {
    lo = __vminu2(lo, m[k]);
    hi = __vmaxu2(hi, m[k]);
  }
  const uint32_t low = min(lo & 0xffffu, lo >> 16), high = max(hi & 0xffffu, hi >> 16);
  return low >= kLogitLow && high < kLogitHigh;
}

}  // namespace mxb200
