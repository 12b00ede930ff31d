// Tables over bf16 logits for the softcap kernels. Device-only.
//
// tanh(z / softcap), and for the loss pass exp(softcap * tanh(z / softcap) - softcap), are functions of one bf16 value:
// 65536 inputs at most, of which a chunk of logits meets a few thousand some 67 million times. A CTA therefore evaluates
// them once per |z| in [2^-16, 2^7) into shared memory and then looks them up, with the bits of the direct evaluation
// because the entries are made by it. A division, a tanhf and an expf are about 60 instructions; a lookup is 4 plus a
// shared-memory read whose 32 random addresses take about 3.5 bank cycles. Values outside the range are evaluated
// directly.
#pragma once

#include <cstdint>

#include <cuda_bf16.h>

namespace mxb200 {

constexpr uint32_t kLogitLow = (127 - 16) << 7;  // bf16 bits of 2^-16
constexpr uint32_t kLogitHigh = (127 + 7) << 7;  // bf16 bits of 2^7, exclusive
constexpr uint32_t kLogitEntries = 2 * (kLogitHigh - kLogitLow);

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

// Entry of the low (half 0) or high 16 bits of w: the bits rotated left by one (magnitude, then sign), times 4 bytes, on a
// table laid out as 2 * (magnitude - low) + sign. table_base: the table's shared-memory address - 8 * kLogitLow.
__device__ __forceinline__ float logit_lookup(uint32_t table_base, uint32_t w, int half) {
  const uint32_t twice = __byte_perm(w, 0u, half ? 0x3232 : 0x1010);
  return load_shared_f32(table_base + ((twice >> 13) & 0x3fffcu));
}

// The logit whose entry is number i.
__device__ __forceinline__ float logit_of_entry(uint32_t i) {
  return __uint_as_float(((kLogitLow + (i >> 1)) | ((i & 1u) << 15)) << 16);
}

// Whether every one of the values in 4 packed words has an entry: magnitudes order as unsigned integers.
__device__ __forceinline__ bool logits_in_table(const uint32_t (&w)[4]) {
  uint32_t lo = w[0] & 0x7fff7fffu, hi = lo;
#pragma unroll
  for (int k = 1; k < 4; ++k) {
    const uint32_t m = w[k] & 0x7fff7fffu;
    lo = __vminu2(lo, m);
    hi = __vmaxu2(hi, m);
  }
  const uint32_t low = min(lo & 0xffffu, lo >> 16), high = max(hi & 0xffffu, hi >> 16);
  return low >= kLogitLow && high < kLogitHigh;
}

}  // namespace mxb200
