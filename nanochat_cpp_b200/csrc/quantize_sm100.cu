// MX quantizer for sm_100a: bf16/fp32 -> E4M3 with one E8M0 scale per 32 values, row-wise and column-wise
// (transposed) in one pass over the input. Replaces nanochat-cpp's nanochat_mx_quantize_* kernels
// (src/nanochat/model/fp8/fp8_kernel.cu:197-210, body mx_kernel.cuh:72-107); same bytes, different schedule.
//
// The unit of work is a 128 x 128 tile, which is exactly one 512-byte swizzled scale tile in each layout.
//   row pass:    each thread takes 16 consecutive values (256-bit loads, one for bf16, two for fp32, fully
//                coalesced); the block maximum of 32 values is a 2-lane shuffle (for plain bf16 input the per-thread
//                maximum stays packed bf16x2 and the multiply by the power-of-two scale is the mixed-precision
//                fp32 = bf16 * bf16 multiply-add, which takes the 16-bit halves as they are); 16 E4M3 bytes leave
//                with one 128-bit store (a warp writes 512 contiguous bytes). The loaded values are parked in
//                shared memory in their input type (prologue values are bf16-exact).
//   column pass: each thread owns two adjacent columns x 32 rows, read from shared memory as packed pairs
//                (a warp reads 128 contiguous bytes per row, conflict-free), needs no shuffle, and writes
//                32 contiguous bytes of each transposed row with one 256-bit store (a full DRAM sector).
//   scales:      staged in shared memory in swizzled order and written as 16-byte vectors, 512 bytes per tile.
// Three schedules: one CTA per tile (every input type and prologue; lists of up to one wave), for plain input of more than
// one wave, bf16 and fp32 tensors in one list, persistent CTAs that draw tiles from a counter and bring them in by TMA a
// tile ahead, and the same in three groups around a shared table for the softcap gradient.
// HBM traffic is the algorithmic minimum: every input byte read once, every output byte written once.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "bf16x2_sm100.cuh"
#include "internal.h"
#include "mx_common.cuh"
#include "ptx_sm100.cuh"
#include "softcap_table_sm100.cuh"

namespace mxb200 {

namespace {

constexpr int kTile = 128;
constexpr int kThreads = 256;

enum Prologue : int { kNone = 0, kReluSquare = 1, kReluSquareBwd = 2, kSoftcapGrad = 3 };

// The softcap cross-entropy gradient prologue's inputs (src/nanochat/model/ops/softcap_ce_kernel.cu:118-145): x holds
// the chunk's logits, and per row a target, the log-sum-exp of its capped logits and an upstream scale.
struct SoftcapGrad {
  const int64_t* targets;
  const float* lse;
  const float* grad_scale;
  int64_t grad_scale_stride;
  const int64_t* num_valid;
  int vocab;
  float softcap;
};

struct QuantParams {
  const void* x;
  const void* h;  // relu^2 backward only
  int64_t cols;   // row stride of x (and h), elements
  mxb200_mx_out out, out_t;
  int tiles_c;
  bool floor_rule;
  bool wide_in;     // x is 32-byte aligned
  bool wide_out_t;  // out_t.data and its ld are 32-byte aligned
  SoftcapGrad ce;   // softcap gradient prologue only
};

// d loss_row / d z of one logit, before rounding, from th = tanh(z / softcap): p = softmax of the capped logits. The
// expressions are the reference's (softcap_ce_kernel.cu:49-54), so the compiler contracts them the same way.
__device__ __forceinline__ float softcap_ce_grad(float th, bool is_target, float lse, float softcap, float scale) {
  const float p = expf(softcap * th - lse);
  return (p - (is_target ? 1.f : 0.f)) * (1.f - th * th) * scale;
}

// Two values at a time: one instruction where the scalar form takes two, the same roundings.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// softcap_ce_grad of two logits that are not the target, rounded to packed bf16.
__device__ __forceinline__ uint32_t softcap_ce_grad_pair(float th0, float th1, uint64_t softcap, uint64_t minus_lse,
                                                         uint64_t scale) {
  const uint64_t th = pack_f32x2(th0, th1);
  const uint64_t minus_th = mul_f32x2(th, 0xbf800000bf800000ull);
  const float2 e = unpack_f32x2(fma_f32x2(softcap, th, minus_lse));
  const uint64_t p = pack_f32x2(expf(e.x), expf(e.y));
  const float2 g = unpack_f32x2(mul_f32x2(mul_f32x2(p, fma_f32x2(th, minus_th, 0x3f8000003f800000ull)), scale));
  return pack_bf16x2_rn(g.x, g.y);
}

__device__ __forceinline__ float bf16_round(float v) {
  return __bfloat162float(__float2bfloat16(v));
}

template <int kPro>
__device__ __forceinline__ float prologue(float v, float h) {
  if constexpr (kPro == kReluSquare) {
    const float r = v <= 0.f ? 0.f : v;
    return bf16_round(r * r);
  } else if constexpr (kPro == kReluSquareBwd) {
    return bf16_round(h <= 0.f ? 0.f : v * (2.f * h));
  } else {
    return v;
  }
}

// Input that is read once. Not through the non-coherent path (.nc): the kernel before may write it while this one has begun.
__device__ __forceinline__ uint4 load_u4_stream(const void* p) {
  uint4 r;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}

__device__ __forceinline__ void store_u32x8(void* p, const uint32_t (&w)[8], bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// two floats -> two E4M3 bytes (RNE, saturating), lo in bits 0-7
__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(r) : "f"(lo), "f"(hi));
  return r;
}

__device__ __forceinline__ uint32_t cvt_e4m3x4(float a, float b, float c, float d) {
  return cvt_e4m3x2(a, b) | (cvt_e4m3x2(c, d) << 16);
}

__device__ __forceinline__ void load_u32x8_stream(const void* p, uint32_t (&w)[8], bool wide) {
  if (wide) {
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(p));
  } else {
    const uint4 a = load_u4_stream(p), b = load_u4_stream(static_cast<const unsigned char*>(p) + 16);
    w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
  }
}

// Column pass over a parked 128 x 128 tile: thread = (column pair, 32-row block); reads packed pairs (a warp reads 128
// contiguous bytes per row), writes 32 contiguous bytes of each transposed row and stages the two scale bytes.
template <bool kIn32>
__device__ __forceinline__ void column_pass(const typename std::conditional<kIn32, float, __nv_bfloat16>::type* tile,
                                            const QuantParams& p, int64_t row0, int64_t col0, unsigned char* sc_cols,
                                            int t) {
  const int cp = t & 63, rb = t >> 6;
  uint32_t wlo[8], whi[8];
  int elo, ehi;
  if constexpr (kIn32) {
    float lo[32], hi[32];
    float mlo = 0.f, mhi = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const float2 f = *reinterpret_cast<const float2*>(tile + (rb * 32 + k) * kTile + 2 * cp);
      lo[k] = f.x, hi[k] = f.y;
      mlo = fmaxf(mlo, fabsf(lo[k]));
      mhi = fmaxf(mhi, fabsf(hi[k]));
    }
    elo = mx_exponent(__float_as_uint(mlo), p.floor_rule), ehi = mx_exponent(__float_as_uint(mhi), p.floor_rule);
    const float mullo = __uint_as_float(mx_multiplier_bits(elo)), mulhi = __uint_as_float(mx_multiplier_bits(ehi));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      wlo[k] = cvt_e4m3x4(lo[4 * k] * mullo, lo[4 * k + 1] * mullo, lo[4 * k + 2] * mullo, lo[4 * k + 3] * mullo);
      whi[k] = cvt_e4m3x4(hi[4 * k] * mulhi, hi[4 * k + 1] * mulhi, hi[4 * k + 2] * mulhi, hi[4 * k + 3] * mulhi);
    }
  } else {
    // the two columns stay packed as bf16 pairs: 32 registers instead of 64, absmax on the 16-bit patterns
    uint32_t w[32];
#pragma unroll
    for (int k = 0; k < 32; ++k)
      w[k] = *reinterpret_cast<const uint32_t*>(tile + (rb * 32 + k) * kTile + 2 * cp);
    // four running maxima, so that the chain of dependent instructions is 8 + 2 long instead of 32
    uint32_t m4[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < 32; ++k)
      m4[k & 3] = max_abs_skip_nan_bf16x2(m4[k & 3], w[k]);
    uint32_t m = max_abs_skip_nan_bf16x2(max_abs_skip_nan_bf16x2(m4[0], m4[1]), max_abs_skip_nan_bf16x2(m4[2], m4[3]));
    m &= 0x7fff7fffu;
    elo = mx_exponent((m & 0xffffu) << 16, p.floor_rule), ehi = mx_exponent(m & 0xffff0000u, p.floor_rule);
    const uint16_t mlo = static_cast<uint16_t>(mx_multiplier_bits(elo) >> 16), mhi = static_cast<uint16_t>(mx_multiplier_bits(ehi) >> 16);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      e4m3x4_scaled_fma_split(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3], mlo, mhi, wlo[k], whi[k]);
  }
  unsigned char* dst = static_cast<unsigned char*>(p.out_t.data) + (col0 + 2 * cp) * p.out_t.ld + row0 + rb * 32;
  store_u32x8(dst, wlo, p.wide_out_t);
  store_u32x8(dst + p.out_t.ld, whi, p.wide_out_t);
  sc_cols[mx_scale_tile_offset(2 * cp, rb)] = static_cast<unsigned char>(elo);
  sc_cols[mx_scale_tile_offset(2 * cp + 1, rb)] = static_cast<unsigned char>(ehi);
}

// One 512-byte scale tile per layout leaves shared memory as 16-byte vectors (threads 0-31 rows, 32-63 columns).
__device__ __forceinline__ void write_scale_tiles(const QuantParams& p, int tile_r, int tile_c, const unsigned char* sc_rows,
                                                  const unsigned char* sc_cols, int t) {
  const bool want_rows = p.out.data != nullptr, want_cols = p.out_t.data != nullptr;
  if (t < 32) {
    if (want_rows)
      reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.out.scale) +
                               (static_cast<int64_t>(tile_r) * p.out.scale_tiles + tile_c) * kScaleTileBytes)[t] =
            reinterpret_cast<const uint4*>(sc_rows)[t];
  } else if (t < 64) {
    if (want_cols)
      reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.out_t.scale) +
                               (static_cast<int64_t>(tile_c) * p.out_t.scale_tiles + tile_r) * kScaleTileBytes)[t - 32] =
            reinterpret_cast<const uint4*>(sc_cols)[t - 32];
  }
}

// kIn32: fp32 input (parked as float), else bf16 (parked as bf16).
// Row pass: a thread owns 16 consecutive values of a row (one 256-bit load of bf16), two lanes share a 32-value
// block (one shuffle), 16 E4M3 bytes leave with one 128-bit store (512 contiguous bytes per warp).
// One CTA's work: tile number `tile_index` (row-major over the tensor's 128 x 128 tiles) of the tensor p describes.
template <bool kIn32, int kPro>
__device__ __forceinline__ void quantize_tile(const QuantParams& p, int tile_index) {
  using Park = typename std::conditional<kIn32, float, __nv_bfloat16>::type;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Park* tile = reinterpret_cast<Park*>(smem_raw);                               // [128][128]
  unsigned char* sc_rows = smem_raw + sizeof(Park) * kTile * kTile;             // 512 B, swizzled
  unsigned char* sc_cols = sc_rows + kScaleTileBytes;                           // 512 B, swizzled

  const int t = static_cast<int>(threadIdx.x);
  const int tile_r = tile_index / p.tiles_c, tile_c = tile_index % p.tiles_c;
  const int64_t row0 = static_cast<int64_t>(tile_r) * kTile, col0 = static_cast<int64_t>(tile_c) * kTile;
  const bool want_rows = p.out.data != nullptr, want_cols = p.out_t.data != nullptr;
  grid_dependency_wait();

  // ---- row pass: 128 rows x 8 vectors of 16 values = 1024 vectors, 4 per thread
  constexpr int kIters = kTile * (kTile / 16) / kThreads;
  constexpr int kWords = kIn32 ? 16 : 8;  // 32-bit words of input per 16 values
  uint32_t raw[kIters][kWords];
  uint32_t rawh[kPro == kReluSquareBwd ? kIters : 1][8];
  // all loads first: 4 (bf16) or 8 (fp32) independent 32-byte requests per thread in flight
#pragma unroll
  for (int it = 0; it < kIters; ++it) {
    const int q = it * kThreads + t, r = q >> 3, c = (q & 7) * 16;
    const int64_t i = (row0 + r) * p.cols + col0 + c;
    if constexpr (kIn32) {
      uint32_t lo[8], hi[8];
      load_u32x8_stream(static_cast<const float*>(p.x) + i, lo, p.wide_in);
      load_u32x8_stream(static_cast<const float*>(p.x) + i + 8, hi, p.wide_in);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        raw[it][k] = lo[k], raw[it][8 + k] = hi[k];
    } else {
      load_u32x8_stream(static_cast<const __nv_bfloat16*>(p.x) + i, raw[it], p.wide_in);
      if constexpr (kPro == kReluSquareBwd)
        load_u32x8_stream(static_cast<const __nv_bfloat16*>(p.h) + i, rawh[it], p.wide_in);
    }
  }
#pragma unroll
  for (int it = 0; it < kIters; ++it) {
    const int q = it * kThreads + t, r = q >> 3, c = (q & 7) * 16;
    float v[16];
    uint32_t m_bits;  // bits of this thread's max |v|
    if constexpr (kIn32) {
      float m = 0.f;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        v[k] = __uint_as_float(raw[it][k]);
        m = fmaxf(m, fabsf(v[k]));  // fmaxf drops NaN, as the reference's amax
      }
      m_bits = __float_as_uint(m);
      if (want_cols) {
        float4* dst = reinterpret_cast<float4*>(tile + r * kTile + c);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
      }
    } else {
      if constexpr (kPro != kNone) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          v[2 * k] = __uint_as_float(raw[it][k] << 16);
          v[2 * k + 1] = __uint_as_float(raw[it][k] & 0xffff0000u);
        }
      }
      if constexpr (kPro == kNone) {
        // the packed maximum skips NaN operands, as the reference's fmaxf does
        uint32_t m = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          m = max_abs_skip_nan_bf16x2(m, raw[it][k]);
        m &= 0x7fff7fffu;
        m_bits = max(m & 0xffffu, m >> 16) << 16;
        if (want_cols) {
          uint4* dst = reinterpret_cast<uint4*>(tile + r * kTile + c);
          dst[0] = make_uint4(raw[it][0], raw[it][1], raw[it][2], raw[it][3]);
          dst[1] = make_uint4(raw[it][4], raw[it][5], raw[it][6], raw[it][7]);
        }
      } else {
        float m = 0.f;
        uint32_t pk[8];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          float hv = 0.f;
          if constexpr (kPro == kReluSquareBwd)
            hv = (k & 1) ? __uint_as_float(rawh[it][k >> 1] & 0xffff0000u) : __uint_as_float(rawh[it][k >> 1] << 16);
          v[k] = prologue<kPro>(v[k], hv);
          m = fmaxf(m, fabsf(v[k]));
        }
        m_bits = __float_as_uint(m);
#pragma unroll
        for (int k = 0; k < 8; ++k)  // prologue values are bf16-exact: repack by truncation
          pk[k] = (__float_as_uint(v[2 * k]) >> 16) | (__float_as_uint(v[2 * k + 1]) & 0xffff0000u);
        if (want_cols) {
          uint4* dst = reinterpret_cast<uint4*>(tile + r * kTile + c);
          dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
      }
    }
    if (want_rows) {
      // non-negative float bits order as integers
      m_bits = max(m_bits, __shfl_xor_sync(0xffffffffu, m_bits, 1));
      const int e = mx_exponent(m_bits, p.floor_rule);
      uint4 o;
      if constexpr (!kIn32 && kPro == kNone) {
        // the multiplier is a power of two: the packed bf16 product is exact wherever e4m3 can tell
        const uint16_t mb = static_cast<uint16_t>(mx_multiplier_bits(e) >> 16);
        o.x = e4m3x4_scaled_fma(raw[it][0], raw[it][1], mb, mb);
        o.y = e4m3x4_scaled_fma(raw[it][2], raw[it][3], mb, mb);
        o.z = e4m3x4_scaled_fma(raw[it][4], raw[it][5], mb, mb);
        o.w = e4m3x4_scaled_fma(raw[it][6], raw[it][7], mb, mb);
      } else {
        const float mul = __uint_as_float(mx_multiplier_bits(e));
        o.x = cvt_e4m3x4(v[0] * mul, v[1] * mul, v[2] * mul, v[3] * mul);
        o.y = cvt_e4m3x4(v[4] * mul, v[5] * mul, v[6] * mul, v[7] * mul);
        o.z = cvt_e4m3x4(v[8] * mul, v[9] * mul, v[10] * mul, v[11] * mul);
        o.w = cvt_e4m3x4(v[12] * mul, v[13] * mul, v[14] * mul, v[15] * mul);
      }
      *reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.out.data) + (row0 + r) * p.out.ld + col0 + c) = o;
      if ((t & 1) == 0)
        sc_rows[mx_scale_tile_offset(r, c >> 5)] = static_cast<unsigned char>(e);
    }
  }
  __syncthreads();

  // ---- column pass, then the scales
  if (want_cols) {
    column_pass<kIn32>(tile, p, row0, col0, sc_cols, t);
    __syncthreads();
  }
  write_scale_tiles(p, tile_r, tile_c, sc_rows, sc_cols, t);
}

// ---- streaming forms: persistent CTAs, tiles drawn from a counter and brought in by TMA
//
// The one-shot kernel above holds a tile's loads in registers, so a CTA reads, computes and writes in turn and only
// the other CTAs of its SM overlap with it. Here three CTAs per SM each keep two 32 KB tile buffers: while all threads
// work on one tile out of shared memory (no load or store instruction is spent on the input), the tiled TMA load of
// the next is in flight, marked evict-first in L2 because the input is read once. Tiles are handed out by a counter
// and not by a fixed stride: the CTAs of one SM advance at very different rates (with a fixed stride the first CTA of
// a 6144-tile tensor was done after 32 us and the last after 81), so a fixed share per CTA leaves most of the machine
// waiting for the slowest. Inside the benchmark step this form takes 27.5 us for a 16384 x 1536 activation and 61 us
// for the 16384 x 4608 gradient of the merged QKV, against 28.3 and 66.7 us for the one-shot kernel.
constexpr int kStreamStages = 2;
#define MXB200_STREAM_CTAS_PER_SM 3  // also the kernel's launch bound
constexpr int kStreamCtasPerSm = MXB200_STREAM_CTAS_PER_SM;
constexpr uint32_t kStreamTileBytes = kTile * kTile * 2;
constexpr uint64_t kStreamWaitLimitNs = 2000000000ull;
constexpr uint64_t kStreamDrainLimitNs = 50000000ull;

struct StreamBarriers {
  uint64_t full[kStreamStages];
  int tile_of[kStreamStages];  // the tile whose load completes full[s]; -1 is the stop sign
  int job_of[kStreamStages];   // and the tensor it belongs to
  uint32_t abort_flag;
};

// One pair of words per launch in flight, taken round-robin: the next tile to hand out and the CTAs that have left.
constexpr int kStreamSchedSlots = 256;

// A group is 256 threads with tile buffers, scale staging and barriers of their own; a CTA holds one (plain form, three
// CTAs per SM) or, where the groups share a table, three (softcap form, one CTA per SM).
constexpr size_t kStreamGroupBytes =
      (kStreamStages * kStreamTileBytes + 4 * kScaleTileBytes + sizeof(StreamBarriers) + 127) / 128 * 128;
constexpr int kSoftcapGroups = 3;
constexpr size_t kSoftcapSmemBytes = kSoftcapGroups * kStreamGroupBytes + kLogitEntries * 4;
static_assert(kSoftcapSmemBytes <= 232448, "shared memory per CTA");

}  // namespace

// Non-zero after a bounded wait of the streaming quantizer ran out: 0x40000000 | CTA << 8 | tile in the CTA's walk.
__device__ uint32_t g_quantize_watchdog_word;
__device__ uint32_t g_quantize_sched[2 * kStreamSchedSlots];

namespace {

__device__ __forceinline__ bool stream_wait(uint64_t* bar, uint32_t parity, StreamBarriers* bars, uint64_t limit_ns,
                                            uint32_t site) {
  if (mbar_try_wait(bar, parity))
    return true;
  const uint64_t t0 = global_timer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 63u) == 0) {
      if (*reinterpret_cast<volatile uint32_t*>(&bars->abort_flag) != 0)
        return false;
      if (global_timer_ns() - t0 > limit_ns) {
        *reinterpret_cast<volatile uint32_t*>(&bars->abort_flag) = 1;
        atomicCAS(&g_quantize_watchdog_word, 0u, 0x40000000u | (blockIdx.x << 8) | (site & 0xffu));
        return false;
      }
    }
  }
  return true;
}

// The end of a walk that stopped before its i-th tile. Loads drawn and not taken (a wait gave up) may still land in this
// CTA's shared memory: they get a bounded time before it leaves. The last walker out hands the slot back zeroed.
__device__ __forceinline__ void stream_leave(StreamBarriers* bars, int i, uint32_t* sched, uint32_t walkers) {
  if (*reinterpret_cast<volatile uint32_t*>(&bars->abort_flag) != 0) {
    for (int j = i; j < i + kStreamStages; ++j) {
      const uint64_t t0 = global_timer_ns();
      while (!mbar_try_wait(&bars->full[j % kStreamStages], static_cast<uint32_t>(j / kStreamStages) & 1u))
        if (global_timer_ns() - t0 > kStreamDrainLimitNs)
          break;
    }
  }
  __threadfence();
  if (atomicAdd(&sched[1], 1u) == walkers - 1) {
    sched[0] = 0u;
    sched[1] = 0u;
    __threadfence();
  }
}

// Row pass from a tile in shared memory. A thread owns 16 consecutive values (32 bytes) and reads them as two 16-byte
// vectors; lanes 4-7 of every eight take the upper vector first, so the eight lanes of a request cover all 32 banks.
__device__ __forceinline__ void stream_row_pass(const __nv_bfloat16* tile, const QuantParams& p, int64_t row0,
                                                int64_t col0, unsigned char* sc_rows, int t) {
  constexpr int kIters = kTile * (kTile / 16) / kThreads;
#pragma unroll
  for (int it = 0; it < kIters; ++it) {
    const int q = it * kThreads + t, r = q >> 3, piece = q & 7, c = piece * 16;
    const int swap = piece >> 2;
    const uint4* src = reinterpret_cast<const uint4*>(tile + r * kTile + c);
    const uint4 a = src[swap], b = src[swap ^ 1];
    uint32_t m = max_abs_skip_nan_bf16x2(
          max_abs_skip_nan_bf16x2(max_abs_skip_nan_bf16x2(a.x, a.y), max_abs_skip_nan_bf16x2(a.z, a.w)),
          max_abs_skip_nan_bf16x2(max_abs_skip_nan_bf16x2(b.x, b.y), max_abs_skip_nan_bf16x2(b.z, b.w)));
    m = max_abs_skip_nan_bf16x2(m, 0u);  // a lone NaN operand gives way to the zero, as in a running maximum from 0
    m &= 0x7fff7fffu;
    uint32_t m_bits = max(m & 0xffffu, m >> 16) << 16;
    m_bits = max(m_bits, __shfl_xor_sync(0xffffffffu, m_bits, 1));
    const int e = mx_exponent(m_bits, p.floor_rule);
    const uint16_t mb = static_cast<uint16_t>(mx_multiplier_bits(e) >> 16);
    const uint32_t a0 = e4m3x4_scaled_fma(a.x, a.y, mb, mb), a1 = e4m3x4_scaled_fma(a.z, a.w, mb, mb);
    const uint32_t b0 = e4m3x4_scaled_fma(b.x, b.y, mb, mb), b1 = e4m3x4_scaled_fma(b.z, b.w, mb, mb);
    const uint4 o = swap ? make_uint4(b0, b1, a0, a1) : make_uint4(a0, a1, b0, b1);
    *reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.out.data) + (row0 + r) * p.out.ld + col0 + c) = o;
    if ((t & 1) == 0)
      sc_rows[mx_scale_tile_offset(r, c >> 5)] = static_cast<unsigned char>(e);
  }
}

// Eight logits (4 packed words) that the table path does not take: outside the table's range, beyond the vocabulary
// (`left` of them are inside) or holding the target (number `hit`). Out of line: it is rare, and eight evaluations of
// tanh inlined at every use push the row pass out of the instruction cache.
__device__ __noinline__ uint4 softcap_grad_direct(uint4 z, int left, int hit, float lse, float softcap, float scale) {
  uint32_t w[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float g[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float v = i != 0 ? hi_f32(w[k]) : lo_f32(w[k]);
      const float th = v == 0.f ? 0.f : softcap_tanh(v, softcap);
      g[i] = 2 * k + i < left ? softcap_ce_grad(th, 2 * k + i == hit, lse, softcap, scale) : 0.f;
    }
    w[k] = pack_bf16x2_rn(g[0], g[1]);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Row pass of the softcap form: the logits of the tile become the loss's gradient, rounded to bf16 as the reference's grad
// kernel would have written it (0 for ignored rows and for the padding columns), in place for the column pass, and leave
// quantized row-wise. tanh comes from the CTA's table (softcap_table_sm100.cuh); what is left per logit is one exp, and two
// and a half instructions for the rest (four without the paired form). The two passes of a 32-row quarter belong to the same
// 64 threads, so that only these wait for one another in between. 2048 x 32768: 98 us (102.6 with scalar arithmetic, sign in
// the table's index and a barrier of the whole group); issue slots 62% used, the path to L1 and shared memory 58%.
__device__ __forceinline__ void stream_row_pass_softcap(__nv_bfloat16* tile, const QuantParams& p, int64_t row0,
                                                        int64_t col0, unsigned char* sc_rows, const float* table,
                                                        int t) {
  constexpr int kIters = kTile * (kTile / 16) / kThreads;
  const int piece = t & 7, c = piece * 16, swap = piece >> 2;
  const int first_row = (t >> 6) * 32 + ((t & 63) >> 3);  // a quarter of the group takes the 32 rows its column pass reads
  const bool want_rows = p.out.data != nullptr;
  const int64_t gcol = col0 + c;
  const int left = static_cast<int>(p.ce.vocab - gcol < 0 ? 0 : (p.ce.vocab - gcol > 16 ? 16 : p.ce.vocab - gcol));
  int64_t target[kIters];
  float lse[kIters], scale[kIters];
#pragma unroll
  for (int it = 0; it < kIters; ++it) {
    const int64_t grow = row0 + first_row + it * 8;
    target[it] = p.ce.targets[grow];
    lse[it] = p.ce.lse[grow];
    scale[it] = p.ce.grad_scale != nullptr ? p.ce.grad_scale[grow * p.ce.grad_scale_stride] : 1.f;
  }
  const float valid = p.ce.num_valid != nullptr ? static_cast<float>(*p.ce.num_valid) : 1.f;
  const uint64_t softcap2 = pack_f32x2(p.ce.softcap, p.ce.softcap);
  const float one_over_valid = 1.f / valid;  // the scale of every row without an upstream gradient
#pragma unroll
  for (int it = 0; it < kIters; ++it) {
    const int r = first_row + it * 8;
    uint4* cell = reinterpret_cast<uint4*>(tile + r * kTile + c);
    const uint4 v0 = cell[swap], v1 = cell[swap ^ 1];
    uint32_t w[2][4] = {{v0.x, v0.y, v0.z, v0.w}, {v1.x, v1.y, v1.z, v1.w}};  // columns c + 8 swap.., c + 8 (swap ^ 1)..
    if (target[it] < 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        w[k >> 2][k & 3] = 0u;
    } else {
      const float s = p.ce.grad_scale == nullptr ? one_over_valid : scale[it] / valid;
      const uint64_t minus_lse2 = pack_f32x2(-lse[it], -lse[it]), s2 = pack_f32x2(s, s);
      const int64_t off = target[it] - gcol;
      const int hit = off >= 0 && off < 16 ? static_cast<int>(off) : -1;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int first = 8 * (swap ^ h);  // of these 8 columns, within the thread's 16
        uint32_t m[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          m[k] = w[h][k] & 0x7fff7fffu;
        if (left - first >= 8 && hit >> 3 != (swap ^ h) && magnitudes_in_table(m)) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            w[h][k] = softcap_ce_grad_pair(logit_tanh(table, w[h][k], m[k], 0), logit_tanh(table, w[h][k], m[k], 1), softcap2,
                                           minus_lse2, s2);
        } else {
          const uint4 g = softcap_grad_direct(make_uint4(w[h][0], w[h][1], w[h][2], w[h][3]), left - first,
                                              hit >> 3 == (swap ^ h) ? hit & 7 : -1, lse[it], p.ce.softcap, s);
          w[h][0] = g.x, w[h][1] = g.y, w[h][2] = g.z, w[h][3] = g.w;
        }
      }
    }
    cell[swap] = make_uint4(w[0][0], w[0][1], w[0][2], w[0][3]);
    cell[swap ^ 1] = make_uint4(w[1][0], w[1][1], w[1][2], w[1][3]);
    if (want_rows) {
      uint32_t m = 0u;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        m = max_abs_skip_nan_bf16x2(m, w[k >> 2][k & 3]);
      m &= 0x7fff7fffu;
      uint32_t m_bits = max(m & 0xffffu, m >> 16) << 16;
      m_bits = max(m_bits, __shfl_xor_sync(0xffffffffu, m_bits, 1));
      const int e = mx_exponent(m_bits, p.floor_rule);
      const uint16_t mb = static_cast<uint16_t>(mx_multiplier_bits(e) >> 16);
      const uint32_t a0 = e4m3x4_scaled_fma(w[0][0], w[0][1], mb, mb), a1 = e4m3x4_scaled_fma(w[0][2], w[0][3], mb, mb);
      const uint32_t b0 = e4m3x4_scaled_fma(w[1][0], w[1][1], mb, mb), b1 = e4m3x4_scaled_fma(w[1][2], w[1][3], mb, mb);
      const uint4 o = swap ? make_uint4(b0, b1, a0, a1) : make_uint4(a0, a1, b0, b1);
      *reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.out.data) + (row0 + r) * p.out.ld + col0 + c) = o;
      if ((t & 1) == 0)
        sc_rows[mx_scale_tile_offset(r, c >> 5)] = static_cast<unsigned char>(e);
    }
  }
}

// The 256 threads of one group: a barrier of their own, and one that tells all of them whether every one said yes.
__device__ __forceinline__ void group_sync(int bar) {
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kThreads) : "memory");
}

// The 64 threads of a group's quarter, which take the same 32 rows of a tile in both passes.
__device__ __forceinline__ void quarter_sync(int bar) {
  asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool group_all(int bar, bool yes) {
  int all;
  asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\tselp.s32 %0, 1, 0, q;\n\t}\n"
        : "=r"(all)
        : "r"(static_cast<int>(yes)), "r"(bar), "n"(kThreads)
        : "memory");
  return all != 0;
}

struct StreamParams {
  QuantParams q;
  int tiles;
  int slot;
};

__device__ __forceinline__ void quantize_stream_softcap(const CUtensorMap* map_x, const StreamParams& sp) {
  constexpr int kGroups = kSoftcapGroups;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int group = static_cast<int>(threadIdx.x) / kThreads;
  const int t = static_cast<int>(threadIdx.x) % kThreads;
  unsigned char* buffers = smem_raw + group * kStreamGroupBytes;
  unsigned char* sc = buffers + kStreamStages * kStreamTileBytes;  // [2 tiles in turn][rows, columns][512]
  StreamBarriers* bars = reinterpret_cast<StreamBarriers*>(sc + 4 * kScaleTileBytes);
  const QuantParams& p = sp.q;
  uint32_t* sched = g_quantize_sched + 2 * sp.slot;  // [0] next tile to hand out, [1] groups that have left
  const uint32_t walkers = gridDim.x * kGroups;      // groups go round the SMs before an SM gets its second

  if (t == 0) {
    for (int s = 0; s < kStreamStages; ++s)
      mbar_init(&bars->full[s], 1);
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  float* table = reinterpret_cast<float*>(smem_raw + kGroups * kStreamGroupBytes);
  for (uint32_t i = threadIdx.x; i < kLogitEntries; i += kThreads * kGroups)
    table[i] = softcap_tanh(__uint_as_float((kLogitLow + i) << 16), p.ce.softcap);
  __syncthreads();
  grid_dependency_wait();

  // Thread 0 posts this CTA's i-th tile and starts its load into buffer i % stages. A number past the last tile is the
  // stop sign: posted once (a bare arrival completes the phase), after which nothing more is drawn or posted.
  // A CTA's first tile is its own number, so its first load does not wait for an atomic; every later tile comes from
  // the launch's counter, which starts at gridDim.x, and each draw is issued a whole tile before its number is needed
  // (the second tile's at the very start, behind the first load). Only one tile is fixed because a CTA may start late:
  // when another kernel (a collective on a side stream) holds SMs, the CTAs that do not fit wait until others have run
  // out of tiles, and whatever is fixed to them is then worked on after everything else.
  bool drawing = true;
  auto post = [&](int i, int tile) {
    const int s = i % kStreamStages;
    if (tile >= sp.tiles) {
      bars->tile_of[s] = -1;
      mbar_arrive(&bars->full[s]);
      drawing = false;
      return;
    }
    bars->tile_of[s] = tile;
    mbar_arrive_expect_tx(1u, &bars->full[s], kStreamTileBytes);
    tma_load_2d_hint(1u, buffers + s * kStreamTileBytes, map_x, &bars->full[s], (tile % p.tiles_c) * kTile,
                     (tile / p.tiles_c) * kTile, l2_policy_evict_first());
  };
  if (t == 0) {
    post(0, static_cast<int>(blockIdx.x + group * gridDim.x));
    for (int i = 1; i < kStreamStages && drawing; ++i)
      post(i, static_cast<int>(walkers + atomicAdd(&sched[0], 1u)));
  }

  int i = 0;
  for (;; ++i) {
    const int s = i % kStreamStages;
    int drawn = 0;  // thread 0: the tile of iteration i + stages, asked for now and posted after this tile
    if (t == 0 && drawing)
      drawn = static_cast<int>(walkers + atomicAdd(&sched[0], 1u));
    const bool landed = stream_wait(&bars->full[s], static_cast<uint32_t>(i / kStreamStages) & 1u, bars,
                                    kStreamWaitLimitNs, static_cast<uint32_t>(i));
    const int tile = landed ? *reinterpret_cast<volatile int*>(&bars->tile_of[s]) : -1;
    if (!group_all(1 + group, tile >= 0))
      break;  // the passes meet at a barrier below: the group goes in together or not at all
    const int tile_r = tile / p.tiles_c, tile_c = tile % p.tiles_c;
    const int64_t row0 = static_cast<int64_t>(tile_r) * kTile, col0 = static_cast<int64_t>(tile_c) * kTile;
    __nv_bfloat16* buf = reinterpret_cast<__nv_bfloat16*>(buffers + s * kStreamTileBytes);
    unsigned char* sc_rows = sc + (i & 1) * 2 * kScaleTileBytes;
    unsigned char* sc_cols = sc_rows + kScaleTileBytes;
    stream_row_pass_softcap(buf, p, row0, col0, sc_rows, table, t);
    fence_proxy_async_smem();  // these writes come before the load that reuses the buffer
    quarter_sync(1 + kGroups + group * 4 + (t >> 6));
    if (p.out_t.data != nullptr)
      column_pass<false>(buf, p, row0, col0, sc_cols, t);
    group_sync(1 + group);  // every thread is done with the buffer and the scale bytes are staged
    if (t == 0 && drawing)
      post(i + kStreamStages, drawn);
    // the next tile stages its scale bytes in the other half, and the one after that comes after another barrier
    write_scale_tiles(p, tile_r, tile_c, sc_rows, sc_cols, t);
  }
  if (t == 0)
    stream_leave(bars, i, sched, walkers);
}

// ---- plain input, one or several tensors: the streaming form over a list of tensors
//
// A stage holds 32 KB of input: a whole 128 x 128 tile of bf16, or the upper or lower 64 rows of a tile of fp32 (half of
// its scale tiles: 8 of every 16 bytes row-wise, 2 of every 4 column-wise). Both kinds may be in one list, so what a
// Linear quantizes together (activation and fp32 weight) is one launch.
struct StreamJob {
  mxb200_mx_out out, out_t;
  int tiles_c;
  int first_unit;
  bool f32, wide_out_t;
};

// What a layer quantizes together, and what a model's weights take (kernel parameters: 1 and 15 KB).
constexpr int kFewJobs = 4, kManyJobs = 64;

template <int kMaxJobs>
struct StreamBatch {
  CUtensorMap maps[kMaxJobs];
  StreamJob jobs[kMaxJobs];
  int n, units, slot;
  bool floor_rule;
};

// fp32 row pass over 64 rows in shared memory: a thread owns 16 consecutive values, read as four 16-byte vectors in an
// order rotated by its pair of lanes, so that the eight lanes of a request cover all 32 banks.
__device__ __forceinline__ void stream_row_pass_f32(const float* tile, const QuantParams& p, int64_t row0, int64_t col0,
                                                    int half, unsigned char* sc_rows, int t) {
  constexpr int kIters = (kTile / 2) * (kTile / 16) / kThreads;
#pragma unroll
  for (int it = 0; it < kIters; ++it) {
    const int q = it * kThreads + t, r = q >> 3, piece = q & 7, c = piece * 16, rot = (piece >> 1) & 3;
    const float4* src = reinterpret_cast<const float4*>(tile + r * kTile + c);
    float4 v[4];
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = src[(i + rot) & 3];
      m = fmaxf(fmaxf(fmaxf(m, fabsf(v[i].x)), fmaxf(fabsf(v[i].y), fabsf(v[i].z))), fabsf(v[i].w));  // drops NaN
    }
    uint32_t m_bits = __float_as_uint(m);
    m_bits = max(m_bits, __shfl_xor_sync(0xffffffffu, m_bits, 1));
    const int e = mx_exponent(m_bits, p.floor_rule);
    const float mul = __uint_as_float(mx_multiplier_bits(e));
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      o[i] = cvt_e4m3x4(v[i].x * mul, v[i].y * mul, v[i].z * mul, v[i].w * mul);
    // o[i] belongs at word (i + rot) & 3
    const bool one = (rot & 1) != 0, two = (rot & 2) != 0;
    const uint32_t a0 = one ? o[3] : o[0], a1 = one ? o[0] : o[1], a2 = one ? o[1] : o[2], a3 = one ? o[2] : o[3];
    *reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.out.data) + (row0 + r) * p.out.ld + col0 + c) =
          two ? make_uint4(a2, a3, a0, a1) : make_uint4(a0, a1, a2, a3);
    if ((t & 1) == 0)
      sc_rows[mx_scale_tile_offset(half * 64 + r, c >> 5)] = static_cast<unsigned char>(e);
  }
}

// fp32 column pass over 64 rows: a thread owns one column of a 32-row block (a warp reads 128 contiguous bytes per row).
__device__ __forceinline__ void stream_column_pass_f32(const float* tile, const QuantParams& p, int64_t row0,
                                                       int64_t col0, int half, unsigned char* sc_cols, int t) {
  const int c = t & (kTile - 1), rb = t >> 7;
  float v[32];
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    v[k] = tile[(rb * 32 + k) * kTile + c];
    m = fmaxf(m, fabsf(v[k]));
  }
  const int e = mx_exponent(__float_as_uint(m), p.floor_rule);
  const float mul = __uint_as_float(mx_multiplier_bits(e));
  uint32_t w[8];
#pragma unroll
  for (int k = 0; k < 8; ++k)
    w[k] = cvt_e4m3x4(v[4 * k] * mul, v[4 * k + 1] * mul, v[4 * k + 2] * mul, v[4 * k + 3] * mul);
  store_u32x8(static_cast<unsigned char*>(p.out_t.data) + (col0 + c) * p.out_t.ld + row0 + rb * 32, w, p.wide_out_t);
  sc_cols[mx_scale_tile_offset(c, half * 2 + rb)] = static_cast<unsigned char>(e);
}

// This half's bytes of the two scale tiles.
__device__ __forceinline__ void write_half_scale_tiles(const QuantParams& p, int tile_r, int tile_c, int half,
                                                       const unsigned char* sc_rows, const unsigned char* sc_cols, int t) {
  if (t < 32) {
    if (p.out.data != nullptr) {
      const int at = t * 16 + half * 8;
      *reinterpret_cast<uint2*>(static_cast<unsigned char*>(p.out.scale) +
                                (static_cast<int64_t>(tile_r) * p.out.scale_tiles + tile_c) * kScaleTileBytes + at) =
            *reinterpret_cast<const uint2*>(sc_rows + at);
    }
  } else if (t >= 128) {
    if (p.out_t.data != nullptr) {
      const int at = (t - 128) * 4 + half * 2;
      *reinterpret_cast<uint16_t*>(static_cast<unsigned char*>(p.out_t.scale) +
                                   (static_cast<int64_t>(tile_c) * p.out_t.scale_tiles + tile_r) * kScaleTileBytes + at) =
            *reinterpret_cast<const uint16_t*>(sc_cols + at);
    }
  }
}

template <int kMaxJobs>
__device__ __forceinline__ void quantize_stream_batch(const StreamBatch<kMaxJobs>& b) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* sc = smem_raw + kStreamStages * kStreamTileBytes;  // [2 units in turn][rows, columns][512]
  StreamBarriers* bars = reinterpret_cast<StreamBarriers*>(sc + 4 * kScaleTileBytes);
  const int t = static_cast<int>(threadIdx.x);
  uint32_t* sched = g_quantize_sched + 2 * b.slot;

  if (t == 0) {
    for (int s = 0; s < kStreamStages; ++s)
      mbar_init(&bars->full[s], 1);
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();
  grid_dependency_wait();

  // as in the softcap form: the first unit is the CTA's own number, later ones are drawn a whole unit ahead
  bool drawing = true;
  auto post = [&](int i, int unit) {
    const int s = i % kStreamStages;
    if (unit >= b.units) {
      bars->tile_of[s] = -1;
      mbar_arrive(&bars->full[s]);
      drawing = false;
      return;
    }
    int lo = 0, hi = b.n;  // the tensor whose units include this one
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (unit >= b.jobs[mid].first_unit)
        lo = mid;
      else
        hi = mid;
    }
    const StreamJob& job = b.jobs[lo];
    const int u = unit - job.first_unit, tile = job.f32 ? u >> 1 : u;
    bars->tile_of[s] = u;
    bars->job_of[s] = lo;
    mbar_arrive_expect_tx(1u, &bars->full[s], kStreamTileBytes);
    tma_load_2d_hint(1u, smem_raw + s * kStreamTileBytes, &b.maps[lo], &bars->full[s], (tile % job.tiles_c) * kTile,
                     (tile / job.tiles_c) * kTile + (job.f32 ? (u & 1) * (kTile / 2) : 0), l2_policy_evict_first());
  };
  if (t == 0) {
    post(0, static_cast<int>(blockIdx.x));
    for (int i = 1; i < kStreamStages && drawing; ++i)
      post(i, static_cast<int>(gridDim.x + atomicAdd(&sched[0], 1u)));
  }

  int i = 0;
  for (;; ++i) {
    const int s = i % kStreamStages;
    int drawn = 0;
    if (t == 0 && drawing)
      drawn = static_cast<int>(gridDim.x + atomicAdd(&sched[0], 1u));
    // the passes shuffle within a warp: its lanes take them together or not at all, also when some gave up waiting
    const bool landed = __all_sync(0xffffffffu, stream_wait(&bars->full[s], static_cast<uint32_t>(i / kStreamStages) & 1u,
                                                            bars, kStreamWaitLimitNs, static_cast<uint32_t>(i))) != 0;
    const int u = landed ? *reinterpret_cast<volatile int*>(&bars->tile_of[s]) : -1;
    const StreamJob& job = b.jobs[u >= 0 ? *reinterpret_cast<volatile int*>(&bars->job_of[s]) : 0];
    const bool f32 = job.f32;
    const int tile = f32 ? u >> 1 : u, half = u & 1;
    const int tile_r = tile / job.tiles_c, tile_c = tile % job.tiles_c;
    const int64_t row0 = static_cast<int64_t>(tile_r) * kTile + (f32 ? half * (kTile / 2) : 0);
    const int64_t col0 = static_cast<int64_t>(tile_c) * kTile;
    const QuantParams p{nullptr, nullptr, 0, job.out, job.out_t, job.tiles_c, b.floor_rule, false, job.wide_out_t, SoftcapGrad{}};
    const unsigned char* buf = smem_raw + s * kStreamTileBytes;
    unsigned char* sc_rows = sc + (i & 1) * 2 * kScaleTileBytes;
    unsigned char* sc_cols = sc_rows + kScaleTileBytes;
    if (u >= 0) {
      if (f32) {
        if (p.out.data != nullptr)
          stream_row_pass_f32(reinterpret_cast<const float*>(buf), p, row0, col0, half, sc_rows, t);
        if (p.out_t.data != nullptr)
          stream_column_pass_f32(reinterpret_cast<const float*>(buf), p, row0, col0, half, sc_cols, t);
      } else {
        if (p.out.data != nullptr)
          stream_row_pass(reinterpret_cast<const __nv_bfloat16*>(buf), p, row0, col0, sc_rows, t);
        if (p.out_t.data != nullptr)
          column_pass<false>(reinterpret_cast<const __nv_bfloat16*>(buf), p, row0, col0, sc_cols, t);
      }
    }
    if (__syncthreads_and(u >= 0) == 0)
      break;
    if (t == 0 && drawing)
      post(i + kStreamStages, drawn);
    if (f32)
      write_half_scale_tiles(p, tile_r, tile_c, half, sc_rows, sc_cols, t);
    else
      write_scale_tiles(p, tile_r, tile_c, sc_rows, sc_cols, t);
  }
  if (t == 0)
    stream_leave(bars, i, sched, gridDim.x);
}

// Small lists (no more units than the machine holds at once): a CTA per tile, which finds its tensor by its first tile.
constexpr int kMaxBatch = 32;

struct BatchJob {
  const void* x;
  int64_t ld;
  mxb200_mx_out out, out_t;
  int tiles_c;
  int first_tile;
  bool f32, wide_in, wide_out_t;
};

struct BatchParams {
  BatchJob jobs[kMaxBatch];
  int n;
  bool floor_rule;
};

enum InputKinds : int { kAllBf16 = 0, kAllF32 = 1, kMixed = 2 };

template <int kKinds>
__device__ __forceinline__ void quantize_batch_tile(const BatchParams& bp) {
  int j = 0;
  const int tile = static_cast<int>(blockIdx.x);
  while (j + 1 < bp.n && tile >= bp.jobs[j + 1].first_tile)
    ++j;
  const BatchJob& job = bp.jobs[j];
  QuantParams p{job.x,      nullptr,         job.ld, job.out, job.out_t, job.tiles_c, bp.floor_rule,
                job.wide_in, job.wide_out_t, SoftcapGrad{}};
  if (kKinds == kAllF32 || (kKinds == kMixed && job.f32))
    quantize_tile<true, kNone>(p, tile - job.first_tile);
  else
    quantize_tile<false, kNone>(p, tile - job.first_tile);
}

}  // namespace
}  // namespace mxb200

// Kernels: global, non-template, plain mxb200_* names, as nanochat-cpp names its own
// (src/nanochat/model/fp8/fp8_kernel.cu:174-175, 197-210). CTAs per SM: four for bf16 input, fewer where a prologue or
// fp32 input needs more registers or shared memory per CTA.
#define MXB200_QUANTIZE_KERNEL(name, IN32, PRO, CTAS)                                                                  \
  __global__ void __launch_bounds__(mxb200::kThreads, CTAS) name(const mxb200::QuantParams p) {                        \
    mxb200::quantize_tile<IN32, PRO>(p, static_cast<int>(blockIdx.x));                                                 \
  }
#define MXB200_QUANTIZE_BATCH_KERNEL(name, KINDS, CTAS)                                                                \
  __global__ void __launch_bounds__(mxb200::kThreads, CTAS) name(const __grid_constant__ mxb200::BatchParams bp) {     \
    mxb200::quantize_batch_tile<KINDS>(bp);                                                                            \
  }
#define MXB200_QUANTIZE_STREAM_KERNEL(name, JOBS)                                                                      \
  __global__ void __launch_bounds__(mxb200::kThreads, MXB200_STREAM_CTAS_PER_SM)                                       \
        name(const __grid_constant__ mxb200::StreamBatch<JOBS> batch) {                                                \
    mxb200::quantize_stream_batch<JOBS>(batch);                                                                        \
  }

MXB200_QUANTIZE_KERNEL(mxb200_quantize_relu_square, false, mxb200::kReluSquare, 4)
MXB200_QUANTIZE_KERNEL(mxb200_quantize_relu_square_bwd, false, mxb200::kReluSquareBwd, 3)
// Streaming form: persistent, three CTAs per SM, each with two 32 KB tile buffers.
MXB200_QUANTIZE_STREAM_KERNEL(mxb200_quantize_stream, mxb200::kFewJobs)
MXB200_QUANTIZE_STREAM_KERNEL(mxb200_quantize_stream_many, mxb200::kManyJobs)
// A few columns of a matrix (the value-embedding gate reads 12), copied or added; bound by the launch.
__global__ void __launch_bounds__(256) mxb200_columns_bf16(__nv_bfloat16* dst, int64_t dst_ld, const __nv_bfloat16* src,
                                                           int64_t src_ld, int64_t n, int cols, bool add) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  mxb200::grid_dependency_wait();
  if (i >= n)
    return;
  const int64_t r = i / cols, c = i % cols;
  const __nv_bfloat16 v = src[r * src_ld + c];
  __nv_bfloat16* d = dst + r * dst_ld + c;
  *d = add ? __float2bfloat16(__bfloat162float(*d) + __bfloat162float(v)) : v;
}
// Softcap form: one CTA of three groups per SM around one table of tanh.
__global__ void __launch_bounds__(mxb200::kThreads * mxb200::kSoftcapGroups, 1)
    mxb200_quantize_softcap_grad(const __grid_constant__ CUtensorMap map_x, const mxb200::StreamParams sp) {
  mxb200::quantize_stream_softcap(&map_x, sp);
}
MXB200_QUANTIZE_BATCH_KERNEL(mxb200_quantize_batch_bf16, mxb200::kAllBf16, 4)
MXB200_QUANTIZE_BATCH_KERNEL(mxb200_quantize_batch_f32, mxb200::kAllF32, 2)
MXB200_QUANTIZE_BATCH_KERNEL(mxb200_quantize_batch_mixed, mxb200::kMixed, 2)

namespace mxb200 {
namespace {

using QuantKernel = void (*)(QuantParams);

template <int kPro>
constexpr QuantKernel quantize_kernel() {
  return kPro == kReluSquare ? mxb200_quantize_relu_square : mxb200_quantize_relu_square_bwd;
}

int check_out(const mxb200_mx_out& o, int64_t ld_min) {
  if (o.data == nullptr)
    return MXB200_OK;
  if (o.scale == nullptr)
    return MXB200_ERR_NULL;
  if (o.ld < ld_min || o.scale_tiles < ld_min / 128)
    return MXB200_ERR_SHAPE;
  if (!aligned16(o.data) || !aligned16(o.scale) || o.ld % 16 != 0)
    return MXB200_ERR_ALIGNMENT;
  return MXB200_OK;
}

template <int kPro>
int launch(const QuantParams& p, int64_t tiles, cudaStream_t stream) {
  constexpr size_t smem = 2 * kTile * kTile + 2 * kScaleTileBytes;
  return launch_kernel(quantize_kernel<kPro>(), static_cast<unsigned>(tiles), kThreads, smem, stream, p);
}

// (rows, ld) row-major, a box of one stage: 128 x 128 of bf16 or 64 x 128 of fp32.
int make_input_map(CUtensorMap* map, const void* x, bool f32, int64_t rows, int64_t cols, int64_t ld) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr)
    return MXB200_ERR_DRIVER;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * (f32 ? 4 : 2)};
  const cuuint32_t box[2] = {kTile, f32 ? kTile / 2 : kTile};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                        const_cast<void*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? MXB200_OK : MXB200_ERR_DRIVER;
}

template <typename Kernel>
int configure_once(Kernel kernel, size_t smem, std::atomic<int>& configured_for) {
  int device = 0;
  cudaGetDevice(&device);
  if (configured_for.load() != device) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess)
      return MXB200_ERR_LAUNCH;
    configured_for.store(device);
  }
  return MXB200_OK;
}

int next_stream_slot() {
  static std::atomic<uint32_t> next_slot{0};
  return static_cast<int>(next_slot.fetch_add(1) % kStreamSchedSlots);
}

int launch_softcap(const QuantParams& p, int64_t rows, int64_t cols, int64_t tiles, int sms, cudaStream_t stream) {
  CUtensorMap map;
  if (int s = make_input_map(&map, p.x, false, rows, cols, p.cols); s != MXB200_OK)
    return s;
  static std::atomic<int> configured_for{-1};
  if (int s = configure_once(mxb200_quantize_softcap_grad, kSoftcapSmemBytes, configured_for); s != MXB200_OK)
    return s;
  const StreamParams sp{p, static_cast<int>(tiles), next_stream_slot()};
  return launch_kernel(mxb200_quantize_softcap_grad, static_cast<unsigned>(std::min<int64_t>(tiles, sms)),
                       kThreads * kSoftcapGroups, kSoftcapSmemBytes, stream, map, sp);
}

using Item = mxb200_quantize_item;

// A caller's list from some member on: of items, or of jobs of one input type.
struct ItemList {
  const Item* items;
  const mxb200_quantize_job* jobs;
  int32_t x_bf16;
  Item operator[](int i) const { return items != nullptr ? items[i] : Item{jobs[i], x_bf16}; }
  ItemList from(int i) const {
    return {items != nullptr ? items + i : nullptr, jobs != nullptr ? jobs + i : nullptr, x_bf16};
  }
};

bool asked(const Item& i) {
  return i.job.out.data != nullptr || i.job.out_t.data != nullptr;
}

int64_t tiles_of(const Item& i) {
  return (i.job.rows / kTile) * (i.job.cols / kTile);
}

bool wide_out_t(const mxb200_mx_out& o) {
  return (reinterpret_cast<uintptr_t>(o.data) & 31u) == 0 && o.ld % 32 == 0;
}

template <int kMaxJobs>
constexpr auto stream_kernel() {
  if constexpr (kMaxJobs == kFewJobs)
    return mxb200_quantize_stream;
  else
    return mxb200_quantize_stream_many;
}

// Streams up to kMaxJobs of the items, from the front; `taken`: how many it went over.
template <int kMaxJobs>
int launch_stream(const ItemList& items, int n, int* taken, bool floor_rule, int sms, cudaStream_t stream) {
  constexpr auto kernel = stream_kernel<kMaxJobs>();
  static std::atomic<int> configured_for{-1};
  if (int s = configure_once(kernel, kStreamGroupBytes, configured_for); s != MXB200_OK)
    return s;
  StreamBatch<kMaxJobs> b;
  b.n = 0;
  int64_t units = 0;
  int i = 0;
  for (; i < n && b.n < kMaxJobs; ++i) {
    const Item it = items[i];
    if (!asked(it))
      continue;
    const bool f32 = it.x_bf16 == 0;
    const int64_t mine = tiles_of(it) * (f32 ? 2 : 1);
    if (units + mine > 0x7fffffffLL)
      break;
    if (int s = make_input_map(&b.maps[b.n], it.job.x, f32, it.job.rows, it.job.cols, it.job.cols); s != MXB200_OK)
      return s;
    b.jobs[b.n++] = StreamJob{it.job.out, it.job.out_t, static_cast<int>(it.job.cols / kTile), static_cast<int>(units), f32,
                              wide_out_t(it.job.out_t)};
    units += mine;
  }
  *taken = i;
  if (b.n == 0)
    return MXB200_OK;
  b.units = static_cast<int>(units);
  b.slot = next_stream_slot();
  b.floor_rule = floor_rule;
  const int64_t most = kStreamCtasPerSm * static_cast<int64_t>(sms);
  return launch_kernel(kernel, static_cast<unsigned>(std::min<int64_t>(units, most)), kThreads, kStreamGroupBytes, stream, b);
}

template <int kKinds>
int launch_batch(const BatchParams& bp, int tiles, cudaStream_t stream) {
  constexpr auto kernel = kKinds == kAllBf16 ? mxb200_quantize_batch_bf16
                          : kKinds == kAllF32 ? mxb200_quantize_batch_f32 : mxb200_quantize_batch_mixed;
  constexpr size_t smem = (kKinds == kAllBf16 ? 2 : 4) * kTile * kTile + 2 * kScaleTileBytes;
  static std::atomic<int> configured_for{-1};
  if (int s = configure_once(kernel, smem, configured_for); s != MXB200_OK)
    return s;
  return launch_kernel(kernel, static_cast<unsigned>(tiles), kThreads, smem, stream, bp);
}

// No prologue: any mix of bf16 and fp32 tensors, all checked.
// More input than the CTA-per-tile form holds at once (four CTAs per SM of bf16 tiles, two of fp32) streams through
// persistent CTAs: those forms would run in several waves, each reading, computing and writing in turn. Below that the
// CTA-per-tile form starts sooner: it needs no tensor map, no draw and no barrier before its first load.
int quantize_items(const ItemList& items, int n, bool floor_rule, const DeviceInfo& dev, cudaStream_t stream) {
  int64_t stages = 0;
  bool bf16 = false, f32 = false;
  for (int i = 0; i < n; ++i) {
    const Item it = items[i];
    if (!asked(it))
      continue;
    stages += tiles_of(it) * (it.x_bf16 != 0 ? 1 : 2);
    (it.x_bf16 != 0 ? bf16 : f32) = true;
  }
  int i = 0;
  if (stages > 4 * static_cast<int64_t>(dev.sms)) {
    while (i < n) {
      int taken = 0;
      const int st = n - i <= kFewJobs ? launch_stream<kFewJobs>(items.from(i), n - i, &taken, floor_rule, dev.sms, stream)
                                       : launch_stream<kManyJobs>(items.from(i), n - i, &taken, floor_rule, dev.sms, stream);
      if (st != MXB200_OK)
        return st;
      i += taken;
    }
    return MXB200_OK;
  }
  while (i < n) {
    BatchParams bp{};
    bp.floor_rule = floor_rule;
    int tiles = 0;
    for (; i < n && bp.n < kMaxBatch; ++i) {
      const Item it = items[i];
      if (!asked(it))
        continue;
      bp.jobs[bp.n++] = BatchJob{it.job.x, it.job.cols, it.job.out, it.job.out_t, static_cast<int>(it.job.cols / kTile), tiles,
                                 it.x_bf16 == 0, (reinterpret_cast<uintptr_t>(it.job.x) & 31u) == 0, wide_out_t(it.job.out_t)};
      tiles += static_cast<int>(tiles_of(it));
    }
    if (bp.n == 0)
      break;
    const int st = !f32 ? launch_batch<kAllBf16>(bp, tiles, stream)
                   : !bf16 ? launch_batch<kAllF32>(bp, tiles, stream) : launch_batch<kMixed>(bp, tiles, stream);
    if (st != MXB200_OK)
      return st;
  }
  return MXB200_OK;
}

int quantize(const void* x, const void* h, bool x_bf16, int64_t rows, int64_t cols, mxb200_mx_out out,
             mxb200_mx_out out_t, int pro, int scale_rule, void* stream, const SoftcapGrad* ce = nullptr,
             int64_t ld = 0) {
  DeviceInfo dev;
  if (int s = current_device(&dev); s != MXB200_OK)
    return s;
  if (x == nullptr || (pro == kReluSquareBwd && h == nullptr))
    return MXB200_ERR_NULL;
  const int64_t most_tiles = x_bf16 ? 0x7fffffffLL : 0x3fffffffLL;  // an fp32 tile is two units of a launch
  if (rows <= 0 || cols <= 0 || rows % kTile != 0 || cols % kTile != 0 || rows * cols / (kTile * kTile) > most_tiles)
    return MXB200_ERR_SHAPE;
  if (scale_rule != MXB200_SCALE_REFERENCE && scale_rule != MXB200_SCALE_OCP_FLOOR)
    return MXB200_ERR_ARGUMENT;
  if (pro != kNone && !x_bf16)
    return MXB200_ERR_ARGUMENT;  // prologues read bf16 only, as the reference
  if (!aligned16(x) || (h != nullptr && !aligned16(h)))
    return MXB200_ERR_ALIGNMENT;
  if (int s = check_out(out, cols); s != MXB200_OK)
    return s;
  if (int s = check_out(out_t, rows); s != MXB200_OK)
    return s;
  if (out.data == nullptr && out_t.data == nullptr)
    return MXB200_OK;
  if (ld == 0)
    ld = cols;
  if (ld < cols || ld % 8 != 0)
    return MXB200_ERR_SHAPE;
  QuantParams p{x, h, ld, out, out_t, static_cast<int>(cols / kTile), scale_rule == MXB200_SCALE_OCP_FLOOR,
                (reinterpret_cast<uintptr_t>(x) & 31u) == 0 && ld % 16 == 0,
                (reinterpret_cast<uintptr_t>(out_t.data) & 31u) == 0 && out_t.ld % 32 == 0, SoftcapGrad{}};
  if (ce != nullptr)
    p.ce = *ce;
  const int64_t tiles = (rows / kTile) * (cols / kTile);
  auto* s = static_cast<cudaStream_t>(stream);
  if (pro == kNone) {
    const Item item{{x, rows, cols, out, out_t}, x_bf16 ? 1 : 0};
    return quantize_items({&item, nullptr, 0}, 1, p.floor_rule, dev, s);
  }
  switch (pro) {
    case kReluSquare:
      return launch<kReluSquare>(p, tiles, s);
    case kReluSquareBwd:
      return launch<kReluSquareBwd>(p, tiles, s);
    case kSoftcapGrad:
      return ce != nullptr ? launch_softcap(p, rows, cols, tiles, dev.sms, s) : MXB200_ERR_NULL;
    default:
      return MXB200_ERR_ARGUMENT;
  }
}

int quantize_list(const ItemList& items, int n, int scale_rule, void* stream) {
  DeviceInfo dev;
  if (int s = current_device(&dev); s != MXB200_OK)
    return s;
  if (n < 0 || (n > 0 && items.items == nullptr && items.jobs == nullptr))
    return MXB200_ERR_NULL;
  if (scale_rule != MXB200_SCALE_REFERENCE && scale_rule != MXB200_SCALE_OCP_FLOOR)
    return MXB200_ERR_ARGUMENT;
  // every one is checked before anything is launched
  for (int i = 0; i < n; ++i) {
    const mxb200_quantize_job j = items[i].job;
    if (j.x == nullptr)
      return MXB200_ERR_NULL;
    if (j.rows <= 0 || j.cols <= 0 || j.rows % kTile != 0 || j.cols % kTile != 0 ||
        j.rows * j.cols / (kTile * kTile) > 0x3fffffffLL)
      return MXB200_ERR_SHAPE;
    if (!aligned16(j.x))
      return MXB200_ERR_ALIGNMENT;
    if (int s = check_out(j.out, j.cols); s != MXB200_OK)
      return s;
    if (int s = check_out(j.out_t, j.rows); s != MXB200_OK)
      return s;
  }
  return quantize_items(items, n, scale_rule == MXB200_SCALE_OCP_FLOOR, dev, static_cast<cudaStream_t>(stream));
}

}  // namespace

}  // namespace mxb200

namespace mxb200 {
uint32_t take_quantize_watchdog_word() {
  uint32_t w = 0;
  if (cudaMemcpyFromSymbol(&w, g_quantize_watchdog_word, sizeof(w)) != cudaSuccess)
    return 0;
  if (w != 0) {
    const uint32_t zero = 0;
    cudaMemcpyToSymbol(g_quantize_watchdog_word, &zero, sizeof(zero));
    static const uint32_t zeros[2 * kStreamSchedSlots] = {};
    cudaMemcpyToSymbol(g_quantize_sched, zeros, sizeof(zeros));
  }
  return w;
}
}  // namespace mxb200


namespace mxb200 {
namespace {
int columns(void* dst, int64_t dst_ld, const void* src, int64_t src_ld, int64_t rows, int64_t cols, bool add, void* stream) {
  DeviceInfo dev;
  if (int s = current_device(&dev); s != MXB200_OK)
    return s;
  if (dst == nullptr || src == nullptr)
    return MXB200_ERR_NULL;
  if (rows <= 0 || cols <= 0 || dst_ld < cols || src_ld < cols || (rows * cols + 255) / 256 > 0x7fffffffLL)
    return MXB200_ERR_SHAPE;
  return launch_kernel(mxb200_columns_bf16, static_cast<unsigned>((rows * cols + 255) / 256), 256, 0,
                       static_cast<cudaStream_t>(stream), static_cast<__nv_bfloat16*>(dst), dst_ld,
                       static_cast<const __nv_bfloat16*>(src), src_ld, rows * cols, static_cast<int>(cols), add);
}
}  // namespace
}  // namespace mxb200

extern "C" int mxb200_copy_columns(void* dst, int64_t dst_ld, const void* src, int64_t src_ld, int64_t rows, int64_t cols,
                                   void* stream) {
  return mxb200::columns(dst, dst_ld, src, src_ld, rows, cols, false, stream);
}

extern "C" int mxb200_add_columns(void* dst, int64_t dst_ld, const void* src, int64_t src_ld, int64_t rows, int64_t cols,
                                  void* stream) {
  return mxb200::columns(dst, dst_ld, src, src_ld, rows, cols, true, stream);
}

extern "C" int mxb200_quantize_mx_items(const mxb200_quantize_item* items, int n, int scale_rule, void* stream) {
  return mxb200::quantize_list({items, nullptr, 0}, n, scale_rule, stream);
}

extern "C" int mxb200_quantize_mx_batch(const mxb200_quantize_job* jobs, int n_jobs, int x_bf16, int scale_rule,
                                        void* stream) {
  return mxb200::quantize_list({nullptr, jobs, x_bf16 != 0}, n_jobs, scale_rule, stream);
}

extern "C" int mxb200_quantize_mx(const void* x, int x_bf16, int64_t rows, int64_t cols, mxb200_mx_out out,
                                  mxb200_mx_out out_t, int prologue, int scale_rule, void* stream) {
  if (prologue != MXB200_PROLOGUE_NONE && prologue != MXB200_PROLOGUE_RELU_SQUARE)
    return MXB200_ERR_ARGUMENT;
  return mxb200::quantize(x, nullptr, x_bf16 != 0, rows, cols, out, out_t, prologue, scale_rule, stream);
}

extern "C" int mxb200_quantize_mx_relu_square_bwd(const void* g, const void* h, int64_t rows, int64_t cols,
                                                  mxb200_mx_out out, mxb200_mx_out out_t, int scale_rule,
                                                  void* stream) {
  return mxb200::quantize(g, h, true, rows, cols, out, out_t, mxb200::kReluSquareBwd, scale_rule, stream);
}

extern "C" int mxb200_softcap_ce_grad_mx(const void* logits, int64_t rows, int64_t ld, const int64_t* targets,
                                         const float* lse, int vocab, int padded, float softcap,
                                         const float* grad_scale, int64_t grad_scale_stride, const int64_t* num_valid,
                                         mxb200_mx_out out, mxb200_mx_out out_t, int scale_rule, void* stream) {
  if (targets == nullptr || lse == nullptr)
    return MXB200_ERR_NULL;
  if (vocab <= 0 || vocab > padded || !(softcap > 0.f))
    return MXB200_ERR_ARGUMENT;
  const mxb200::SoftcapGrad ce{targets, lse, grad_scale, grad_scale_stride, num_valid, vocab, softcap};
  return mxb200::quantize(logits, nullptr, true, rows, padded, out, out_t, mxb200::kSoftcapGrad, scale_rule, stream,
                          &ce, ld);
}
