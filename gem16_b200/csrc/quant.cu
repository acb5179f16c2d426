// Activation quantizers: NVFP4 block quantizer (plain, RMSNorm-fused, gated-GELU-fused), the
// compact->interleaved scale shuffle, and the FP8 per-token quantizer (plain, RMSNorm-fused).
//
// All of them are HBM-streaming kernels: every input element is read once with 128-bit loads,
// every output byte written once.  Algorithmic bytes per element (bf16 input): NVFP4
// 2 + 0.5 + 1/16 = 2.5625 B, FP8 2 + 1 = 3 B (+4 B per token).
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace gemb {
namespace {

// Sixteen / eight consecutive elements of a dependent input (an earlier kernel may have written it).
__device__ __forceinline__ void unpack8(const uint4& t, float (&v)[8]) {
  const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[2 * j] = __uint_as_float(w[j] << 16);
    v[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ void load16(const float* p, float (&v)[16]) {
  const float4* q = reinterpret_cast<const float4*>(p);
  float4 t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = ld_dep(q + i);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[4 * i] = t[i].x; v[4 * i + 1] = t[i].y; v[4 * i + 2] = t[i].z; v[4 * i + 3] = t[i].w;
  }
}
__device__ __forceinline__ void load16(const uint16_t* p, float (&v)[16]) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  const uint4 t0 = ld_dep(q), t1 = ld_dep(q + 1);
  float a[8], b[8];
  unpack8(t0, a);
  unpack8(t1, b);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = a[i];
    v[8 + i] = b[i];
  }
}

template <typename In>
struct PlainLoader {
  const In* x;
  __device__ __forceinline__ void operator()(uint64_t offset, float (&v)[16]) const {
    load16(x + offset, v);
  }
};

// src/cuda/nvfp4/reference.cu:177-190.  For fp32 inputs gate/up are first rounded to bf16.
template <typename In>
struct GatedGeluLoader {
  const In* gate;
  const In* up;
  __device__ __forceinline__ void operator()(uint64_t offset, float (&v)[16]) const {
    float g[16], u[16];
    load16(gate + offset, g);
    load16(up + offset, u);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float gv = sizeof(In) == 4 ? bf16_round(g[i]) : g[i];
      const float uv = sizeof(In) == 4 ? bf16_round(u[i]) : u[i];
      v[i] = gelu_tanh_product(gv, uv);
    }
  }
};

// The four scale bytes of a quad (four consecutive 16-blocks, one per lane of an aligned group of four) in one
// word, little end first; every lane of the group gets it.
__device__ __forceinline__ uint32_t quad_scale_word(uint32_t byte) {
  const int pos = threadIdx.x & 3;
  uint32_t w = byte << (8 * pos);
  w |= __shfl_xor_sync(0xFFFFFFFFu, w, 1);
  w |= __shfl_xor_sync(0xFFFFFFFFu, w, 2);
  return w;
}

// One thread per 16-element block: 32 (bf16) or 64 bytes in, 8 payload bytes out, so that a warp's loads
// and stores cover whole lines; four lanes pool their scale bytes into one 32-bit store.  The thread grid
// covers rows_out x blocks_pad where, for the interleaved layout, rows_out is `tokens` rounded up to 128 and
// padded cells get zero scales.  Bound by HBM at prefill sizes (2.56 B per bf16 element); a thread per quad,
// the former split, read 128 bytes per thread with 128-byte strides between lanes and left a one-token call
// with a single CTA.
template <class Loader, bool kRcp, bool kInterleaved>
__global__ void __launch_bounds__(256)
nvfp4_quantize_kernel(Loader loader, uint8_t* __restrict__ packed, uint8_t* __restrict__ scales,
                      uint32_t tokens, uint64_t k, uint32_t blocks_pad, uint64_t cells, float g) {
  pdl_trigger_few_rows(tokens);
  pdl_wait();
  // blockDim and cells are multiples of 4: quads stay whole.  A 64-bit division costs as much as the
  // quantisation of a block, so it is left to tensors that need it.
  const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t r = (cells >> 32) == 0 ? static_cast<uint32_t>(idx) / blocks_pad : idx / blocks_pad;
  const uint32_t c = static_cast<uint32_t>(idx - r * blocks_pad);
  const uint32_t c_real = static_cast<uint32_t>(k / 16);
  const bool live = idx < cells && r < tokens && c < c_real;
  uint8_t sb = 0;
  if (live) {
    float v[16];
    loader(r * k + static_cast<uint64_t>(c) * 16, v);
    uint32_t lo, hi;
    quantize_block16<kRcp>(v, g, lo, hi, sb);
    *reinterpret_cast<uint2*>(packed + r * (k / 2) + static_cast<uint64_t>(c) * 8) = make_uint2(lo, hi);
  }
  const uint32_t word = quad_scale_word(sb);
  if (idx >= cells) return;
  if constexpr (kInterleaved) {
    if ((c & 3) == 0) *reinterpret_cast<uint32_t*>(scales + interleaved_scale_offset(r, c, blocks_pad)) = word;
  } else {
    uint8_t* row = scales + r * c_real;
    if (c_real % 4 == 0) {
      if ((c & 3) == 0) *reinterpret_cast<uint32_t*>(row + c) = word;
    } else if (live) {
      row[c] = sb;
    }
  }
}

template <class Loader>
int32_t launch_nvfp4_quantize(const char* op, Loader loader, uint8_t* packed, uint8_t* scales,
                              uint64_t tokens, uint64_t k, float g, int32_t layout, int32_t mode,
                              cudaStream_t stream) {
  const bool inter = layout == GEMB_SCALES_INTERLEAVED;
  const uint64_t blocks_pad = (k / 16 + 3) / 4 * 4;
  const bool rcp = mode == GEMB_QUANT_RCP_APPROX;
  auto kern = inter ? (rcp ? nvfp4_quantize_kernel<Loader, true, true> : nvfp4_quantize_kernel<Loader, false, true>)
                    : (rcp ? nvfp4_quantize_kernel<Loader, true, false> : nvfp4_quantize_kernel<Loader, false, false>);
  const uint64_t cells = (inter ? (tokens + 127) / 128 * 128 : tokens) * blocks_pad;
  // Few cells (a decode token): small CTAs, so that they spread over the SMs and load side by side.
  const unsigned threads = cells <= 16384 ? 64 : 256;
  GEMB_TRY(launch_pdl_split(op, tokens <= kFewRows, kern, dim3(static_cast<unsigned>((cells + threads - 1) / threads)), dim3(threads), 0, stream,
                            loader, packed, scales, static_cast<uint32_t>(tokens), k, static_cast<uint32_t>(blocks_pad), cells, g));
  return check_launch(op);
}

int32_t validate_nvfp4_quantize(const char* op, const void* in, const void* packed,
                                const void* scales, int32_t dtype, uint64_t tokens, uint64_t k,
                                float g, int32_t layout, int32_t mode) {
  GEMB_REQUIRE(in && packed && scales, "%s: pointers must be nonnull", op);
  GEMB_REQUIRE(dtype == GEMB_F32 || dtype == GEMB_BF16, "%s: input dtype must be GEMB_F32 or GEMB_BF16", op);
  GEMB_REQUIRE(tokens > 0 && k > 0 && k % 16 == 0,
               "%s: extent must be a nonzero multiple of 16 per token", op);
  GEMB_REQUIRE(tokens <= (1ull << 31) && k <= (1ull << 31), "%s: extent too large", op);
  GEMB_REQUIRE(positive_finite(g), "%s: global divisor must be positive and finite", op);
  GEMB_REQUIRE(layout == GEMB_SCALES_COMPACT || layout == GEMB_SCALES_INTERLEAVED, "%s: unknown scale layout", op);
  GEMB_REQUIRE(mode == GEMB_QUANT_EXACT || mode == GEMB_QUANT_RCP_APPROX, "%s: unknown quantizer mode", op);
  GEMB_REQUIRE(reinterpret_cast<uintptr_t>(in) % 16 == 0 && reinterpret_cast<uintptr_t>(packed) % 8 == 0 &&
                   reinterpret_cast<uintptr_t>(scales) % 4 == 0,
               "%s: input must be 16-byte, payload 8-byte and scales 4-byte aligned", op);
  return require_sm100(op);
}

// ---------------------------------------------------------------------------------------------
// Row kernels: RMSNorm fused quantizers, RMSNorm + residual, the FP8 per-token quantizer.
//
// The sum of squares follows the reference exactly: residue t of the row (indices t, t + 256, ...) is one fma
// chain, and a power-of-two tree folds the 256 partials (strides 128, 64, ..., 1;
// src/cuda/nvfp4/reference.cu:102-118), so the fp32 sum is bit-identical.  Both forms below keep that order:
//   warp form   one warp per row.  Lane l holds eight consecutive elements of every 256-element chunk, i.e. the
//               residues 8l .. 8l+7: eight independent chains per lane, the chunks in order, then the tree as
//               shuffles.  The row (bf16, at most 4,096 elements) stays in registers between the passes, so
//               it is read once, with 16-byte loads that are all in flight together, and nothing
//               waits at a CTA barrier.  For batches that give every SM several rows.
//   CTA form    256 threads per row, thread t owns residue t.  For few rows (a decode token: eight warps
//               share the arithmetic of one row), fp32 inputs and long rows.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float sqrt_inverse(float sum, uint64_t k, float eps) {
  return rsqrtf(sum / static_cast<float>(k) + eps);
}
__device__ __forceinline__ float2 bf16x2_to_float2(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
__device__ __forceinline__ uint32_t float2_to_bf16x2(float2 v) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
  return r;
}
// acc += v * v for a bf16 v, one rounding (mixed-precision fma: no unpacking, and off the integer pipe).
__device__ __forceinline__ void fma_bf16(float& acc, uint16_t v) {
  asm("fma.rn.f32.bf16 %0, %1, %1, %0;" : "+f"(acc) : "h"(v));
}
// Larger magnitude per half of two bf16 pairs whose sign bits are already cleared.
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ float max_of_halves(uint32_t w) {
  return fmaxf(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
__device__ __forceinline__ uint32_t abs_max4(const uint32_t (&w)[4]) {
  return max_bf16x2(max_bf16x2(w[0] & 0x7FFF7FFFu, w[1] & 0x7FFF7FFFu), max_bf16x2(w[2] & 0x7FFF7FFFu, w[3] & 0x7FFF7FFFu));
}

constexpr int kRowChunks = 16;       // 256-element chunks a warp keeps in registers
constexpr int kRowWarps = 4;         // rows (warps) per CTA of the warp form
enum { kRowFp8 = 0, kRowFp8Norm = 1, kRowNvfp4Compact = 2, kRowNvfp4Interleaved = 3, kRowResidual = 4 };

struct RowArgs {
  const void* x;
  const uint16_t* w;         // RMSNorm weight, may be null
  uint8_t* out8;             // E4M3 bytes or E2M1 payload
  void* scales;              // fp32 per row (FP8) or E4M3 block scales
  const void* residual;
  float* normalized;
  void* out;                 // RMSNorm + residual
  const uint16_t* scalar;
  uint64_t rows, k;
  float eps, g;
  uint32_t rows_out;         // interleaved scales: rows rounded up to 128 (the padding is written as zero)
};

// Eight normalised elements as bf16 pairs: bf16((x * inv) * w).
__device__ __forceinline__ void normalise8(const uint4& raw, const uint4* w, bool has_w, float inv, uint32_t (&n)[4]) {
  const uint32_t xw[4] = {raw.x, raw.y, raw.z, raw.w};
  uint4 wv = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);   // ones
  if (has_w) wv = __ldg(w);
  const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    n[j] = float2_to_bf16x2(__fmul2_rn(__fmul2_rn(bf16x2_to_float2(xw[j]), make_float2(inv, inv)), bf16x2_to_float2(ww[j])));
}

// Warp form.  bf16 rows, k a multiple of 16 and at most 4,096, 16-byte aligned rows.
// Measured on 16,384 x 3,840 (4,096 for the plain FP8 quantizer), before (one CTA per row: 2-byte loads for the sum,
// eight barriers, every pass from memory again, a division per element) and now, against the bytes at the copy peak:
//   RMSNorm + FP8     184 -> 58 us (29)       FP8            66 -> 36 us (31)
//   RMSNorm + NVFP4   142 -> 66 us (25)       RMSNorm + residual   140 -> 65 us (59)
// The FP8 and residual forms are bound by HBM; the normalising quantizers by the integer pipe (unpacking
// bf16, amax, scale bytes: about nine instructions per element there).
template <int kMode, bool kRcp>
__global__ void __launch_bounds__(kRowWarps * 32, kMode == kRowResidual ? 4 : 5)
row_warp_kernel(const __grid_constant__ RowArgs a) {
  constexpr bool kNorm = kMode != kRowFp8;
  if constexpr (kNorm) pdl_trigger();   // a normalised tensor is no weight
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const uint64_t r = static_cast<uint64_t>(blockIdx.x) * kRowWarps + (threadIdx.x >> 5);
  const uint32_t k = static_cast<uint32_t>(a.k);
  if constexpr (kMode == kRowNvfp4Interleaved) {
    if (r >= a.rows) {   // padding row of the interleaved scale buffer
      const uint32_t quads = (k / 16 + 3) / 4;
      if (r < a.rows_out)
        for (uint32_t q = lane; q < quads; q += 32)
          *reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(a.scales) + interleaved_scale_offset(r, 4 * q, quads * 4)) = 0;
      return;
    }
  } else {
    if (r >= a.rows) return;
  }
  const uint16_t* row = static_cast<const uint16_t*>(a.x) + r * k;
  uint4 raw[kRowChunks];
#pragma unroll
  for (int c = 0; c < kRowChunks; ++c) {
    const uint32_t i = c * 256 + lane * 8;
    raw[c] = make_uint4(0, 0, 0, 0);
    if (i < k) raw[c] = ld_dep(reinterpret_cast<const uint4*>(row + i));
  }
  // The residual's first eight chunks are requested before the reduction, the others behind the first half of the output.
  uint4 res[kMode == kRowResidual ? 8 : 1];
  auto load_residual = [&](int c0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t i = (c0 + u) * 256 + lane * 8;
      if (i < k) res[kMode == kRowResidual ? u : 0] = ld_dep(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(a.residual) + r * k + i));
    }
  };
  if constexpr (kMode == kRowResidual) load_residual(0);
  float inv = 1.0f;
  if constexpr (kNorm) {
    float ss[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) ss[j] = 0.0f;
#pragma unroll
    for (int c = 0; c < kRowChunks; ++c) {
      if (c * 256 >= static_cast<int>(k)) break;   // elements past k are zero and add nothing
      const uint32_t xw[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        fma_bf16(ss[2 * j], static_cast<uint16_t>(xw[j]));
        fma_bf16(ss[2 * j + 1], static_cast<uint16_t>(xw[j] >> 16));
      }
    }
    // Tree over residues 8 * lane + j.  Strides 128, 64, 32 pair lanes 16, 8, 4 apart: each step keeps half of
    // the lane's residues (the lane's bit picks which), so that the later steps carry one value instead of eight.
    float h4[4], h2[2], s;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float mine = (lane & 16) ? ss[4 + j] : ss[j], theirs = (lane & 16) ? ss[j] : ss[4 + j];
      h4[j] = mine + __shfl_xor_sync(0xFFFFFFFFu, theirs, 16);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float mine = (lane & 8) ? h4[2 + j] : h4[j], theirs = (lane & 8) ? h4[j] : h4[2 + j];
      h2[j] = mine + __shfl_xor_sync(0xFFFFFFFFu, theirs, 8);
    }
    s = ((lane & 4) ? h2[1] : h2[0]) + __shfl_xor_sync(0xFFFFFFFFu, (lane & 4) ? h2[0] : h2[1], 4);
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);     // stride 16
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);     // stride 8
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 16);    // strides 4, 2, 1: the residue's low bits sit in lane bits 4, 3, 2
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 8);
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 4);
    inv = sqrt_inverse(s, k, a.eps);
  }
  const bool has_w = a.w != nullptr;
  const uint4* wp = reinterpret_cast<const uint4*>(a.w) + lane;

  if constexpr (kMode == kRowFp8 || kMode == kRowFp8Norm) {
    uint32_t amax2 = 0;
#pragma unroll
    for (int c = 0; c < kRowChunks; ++c) {
      if (c * 256 >= static_cast<int>(k)) break;
      if constexpr (kNorm) {
        uint32_t n[4];
        normalise8(raw[c], wp + c * 32, has_w && c * 256 + lane * 8 < static_cast<int>(k), inv, n);
        raw[c] = make_uint4(n[0], n[1], n[2], n[3]);
      }
      const uint32_t n[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
      amax2 = max_bf16x2(amax2, abs_max4(n));
    }
    const Quotient q = token_quotient(warp_max(max_of_halves(amax2)));
    if (lane == 0) static_cast<float*>(a.scales)[r] = q.scale;
    uint8_t* out = a.out8 + r * k + lane * 8;
    auto convert = [&](auto code) {
#pragma unroll
      for (int c = 0; c < kRowChunks; ++c) {
        if (c * 256 + lane * 8 >= k) break;
        const uint32_t n[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
        uint32_t p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = code(bf16x2_to_float2(n[j]));
        *reinterpret_cast<uint2*>(out + c * 256) = make_uint2(__byte_perm(p[0], p[1], 0x5410), __byte_perm(p[2], p[3], 0x5410));
      }
    };
    if (q.divide) convert([&](float2 v) { return e4m3x2_divided(v.x, v.y, q.scale); });
    else convert([&](float2 v) { return e4m3_of_quotients(v, q); });
  } else if constexpr (kMode == kRowNvfp4Compact || kMode == kRowNvfp4Interleaved) {
    const uint32_t c_real = k / 16, c_pad = (c_real + 3) / 4 * 4;
    // Chunk c covers blocks 16c .. 16c + 15, one per lane pair; addresses advance by constants.
    uint8_t* pay = a.out8 + r * (k / 2) + lane * 4;
    uint8_t* sc = static_cast<uint8_t*>(a.scales);
    if constexpr (kMode == kRowNvfp4Interleaved) sc += interleaved_scale_offset(r, (lane >> 3) * 4, c_pad);
    else sc += r * c_real + (lane >> 1);
#pragma unroll
    for (int c = 0; c < kRowChunks; ++c) {
      if (c * 256 >= static_cast<int>(k)) break;
      const uint32_t i = c * 256 + lane * 8;   // lanes 2b and 2b + 1 share a 16-element block
      uint32_t n[4];
      normalise8(raw[c], wp + c * 32, has_w && i < k, inv, n);
      uint32_t m = abs_max4(n);
      m = max_bf16x2(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
      const BlockScale s = block_scale<kRcp>(max_of_halves(m), a.g);
      uint32_t p[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) p[j] = quantize_pair<kRcp>(bf16x2_to_float2(n[j]), a.g, s);
      uint32_t word = __byte_perm(__byte_perm(p[0], p[1], 0x0040), __byte_perm(p[2], p[3], 0x0040), 0x5410);
      if (!kRcp && s.ds == 0.0f) word = 0;
      if (i < k) *reinterpret_cast<uint32_t*>(pay + c * 128) = word;
      if (kMode == kRowNvfp4Interleaved || c_real % 4 == 0) {
        // four blocks = eight lanes: their scale bytes leave as one word
        uint32_t sw = i < k ? static_cast<uint32_t>(s.bits) << (8 * ((lane >> 1) & 3)) : 0u;
        sw |= __shfl_xor_sync(0xFFFFFFFFu, sw, 2);
        sw |= __shfl_xor_sync(0xFFFFFFFFu, sw, 4);
        if ((lane & 7) == 0 && i / 16 < c_pad)
          *reinterpret_cast<uint32_t*>(sc + c * (kMode == kRowNvfp4Interleaved ? 2048 : 16)) = sw;
      } else if ((lane & 1) == 0 && i < k) {
        sc[c * 16] = s.bits;
      }
    }
  } else {
    const float layer_scale = a.scalar ? bf16_bits_to_float(__ldg(a.scalar)) : 1.0f;
    uint16_t* out = static_cast<uint16_t*>(a.out) + r * k;
#pragma unroll
    for (int c0 = 0; c0 < kRowChunks; c0 += 8) {
      if (c0 != 0) load_residual(c0);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int c = c0 + u;
        const uint32_t i = c * 256 + lane * 8;
        if (i >= k) break;
        const uint32_t rw[4] = {res[u].x, res[u].y, res[u].z, res[u].w};
        uint32_t n[4];
        normalise8(raw[c], wp + c * 32, has_w, inv, n);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          n[j] = float2_to_bf16x2(__fadd2_rn(bf16x2_to_float2(n[j]), bf16x2_to_float2(rw[j])));
          if (a.scalar) n[j] = float2_to_bf16x2(__fmul2_rn(bf16x2_to_float2(n[j]), make_float2(layer_scale, layer_scale)));
        }
        *reinterpret_cast<uint4*>(out + i) = make_uint4(n[0], n[1], n[2], n[3]);
      }
    }
  }
}

// ---- CTA form ---------------------------------------------------------------------------------
__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(uint16_t v) { return bf16_bits_to_float(v); }

// Few rows of up to kShortRow elements are read once: thread t holds elements t, t + 256, ... (the sum's order) in registers
// and, where the second half of the kernel wants sixteen neighbours, hands them over through shared memory.  A decode
// step's row kernels are a chain of memory round trips: norm weights come before the wait for the previous kernel and
// the second read of the row is gone (3,840 elements: RMSNorm + residual 4.0 -> 3.1 us behind its predecessor,
// + FP8 3.3 -> 3.0; a decode pass 231 -> 218 us).
constexpr uint32_t kShortRow = 256 * 16;
// For the few rows of a decode step only: behind a GEMM, which starts nothing early, there is no wait to load weights under, and
// the wider second read is the faster one (77-token layer 72.8 us against 74.3).
bool short_rows(uint64_t rows, uint64_t k) { return k <= kShortRow && rows <= 16; }

// Every warp folds the 256 partials by itself, in the tree's order: strides 128, 64, 32 inside the lane, the
// rest as shuffles.  One barrier instead of eight.
__device__ __forceinline__ float rmsnorm_fold(float ss, uint64_t k, float eps, float* red) {
  red[threadIdx.x] = ss;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  float p[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) p[j] = red[lane + 32 * j];
  float s = ((p[0] + p[4]) + (p[2] + p[6])) + ((p[1] + p[5]) + (p[3] + p[7]));
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
  return sqrt_inverse(s, k, eps);
}

// A short row into registers, its sum of squares in the same order as below.
template <typename In>
__device__ __forceinline__ float load_short_row(const In* row, uint32_t k, float (&v)[16]) {
  In raw[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const uint32_t i = threadIdx.x + j * 256;
    raw[j] = In(0);
    if (i < k) raw[j] = ld_dep(row + i);
  }
  float ss = 0.0f;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    v[j] = to_float(raw[j]);
    ss = fmaf(v[j], v[j], ss);
  }
  return ss;
}
// The norm weights of elements 16 c .. 16 c + 15, before the wait for the previous kernel (they are at rest).
__device__ __forceinline__ void load_norm_weights(const uint16_t* w, uint32_t c, uint32_t k, uint16_t (&wv)[16]) {
  if (w && c * 16 < k && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {   // k is a multiple of 16
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(w) + 2 * c), b = __ldg(reinterpret_cast<const uint4*>(w) + 2 * c + 1);
    const uint32_t words[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 16; ++i) wv[i] = static_cast<uint16_t>(words[i / 2] >> (16 * (i & 1)));
    return;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) wv[i] = w && c * 16 + i < k ? __ldg(w + c * 16 + i) : uint16_t(0x3F80);
}
// 1 / rms of a short row whose elements it leaves in xs.
template <typename In>
__device__ __forceinline__ float stage_short_row(const In* row, uint32_t k, float eps, float* xs, float* red) {
  float v[16];
  const float ss = load_short_row(row, k, v);
#pragma unroll
  for (int j = 0; j < 16; ++j)
    if (threadIdx.x + j * 256 < k) xs[threadIdx.x + j * 256] = v[j];
  return rmsnorm_fold(ss, k, eps, red);   // its barrier covers xs
}
__device__ __forceinline__ void normalise_staged(const float* xs, uint32_t c, const uint16_t (&wv)[16], float inv, float (&v)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 x = *reinterpret_cast<const float4*>(xs + c * 16 + 4 * q);
    v[4 * q] = x.x, v[4 * q + 1] = x.y, v[4 * q + 2] = x.z, v[4 * q + 3] = x.w;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = bf16_round(__fmul_rn(__fmul_rn(v[i], inv), bf16_bits_to_float(wv[i])));
}

template <typename In>
__device__ __forceinline__ float rmsnorm_inverse(const In* row, uint64_t k, float eps, float* red) {
  float ss = 0.0f;
  // sixteen loads of the thread's chain in flight at a time; zeros past the end add nothing
  for (uint64_t base = threadIdx.x; base < k; base += 256 * 16) {
    In raw[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint64_t i = base + j * 256;
      raw[j] = In(0);
      if (i < k) raw[j] = ld_dep(row + i);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float v = to_float(raw[j]);
      ss = fmaf(v, v, ss);
    }
  }
  return rmsnorm_fold(ss, k, eps, red);
}

// RMSNorm + residual (+ layer scalar) with the bf16 boundaries of src/cuda/norm/reference.cu:66-160:
// n = bf16(x * inv * w), v = bf16(n + residual), v = bf16(v * scalar) when a scalar is given.
__device__ __forceinline__ void store_scalar(float* p, uint64_t i, float v) { p[i] = v; }
__device__ __forceinline__ void store_scalar(uint16_t* p, uint64_t i, float v) { p[i] = float_to_bf16_bits(v); }

// Any width and alignment: the second pass takes one element per thread and step, eight steps in flight.
template <typename In, typename Res, typename Out, bool kShort>
__global__ void __launch_bounds__(256)
rmsnorm_residual_kernel(const In* x, const uint16_t* __restrict__ w, const Res* residual, float* normalized, Out* out,
                        uint64_t k, float eps, const uint16_t* __restrict__ scalar) {
  __shared__ float red[256];
  pdl_trigger();
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * k;
  if constexpr (kShort) {
    uint16_t wv[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) wv[j] = w && threadIdx.x + j * 256 < k ? __ldg(w + threadIdx.x + j * 256) : uint16_t(0x3F80);
    const float layer_scale = scalar ? bf16_bits_to_float(__ldg(scalar)) : 1.0f;
    prefetch_l2_span(residual + base, k * sizeof(Res));
    pdl_wait();
    Res rv[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      rv[j] = Res(0);
      if (threadIdx.x + j * 256 < k) rv[j] = ld_dep(residual + base + threadIdx.x + j * 256);
    }
    float xv[16];
    const float ss = load_short_row(x + base, static_cast<uint32_t>(k), xv);
    const float inv = rmsnorm_fold(ss, k, eps, red);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint64_t i = threadIdx.x + j * 256;
      if (i >= k) continue;
      const float n = bf16_round(__fmul_rn(__fmul_rn(xv[j], inv), bf16_bits_to_float(wv[j])));
      if (normalized) normalized[base + i] = n;
      float v = bf16_round(__fadd_rn(n, to_float(rv[j])));
      if (scalar) v = bf16_round(__fmul_rn(v, layer_scale));
      store_scalar(out, base + i, v);
    }
    return;
  }
  pdl_wait();
  const float inv = rmsnorm_inverse(x + base, k, eps, red);
  const float layer_scale = scalar ? bf16_bits_to_float(__ldg(scalar)) : 1.0f;
  for (uint64_t i0 = threadIdx.x; i0 < k; i0 += 256 * 8) {
    In xv[8];
    Res rv[8];
    uint16_t wv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint64_t i = i0 + j * 256;
      if (i >= k) continue;
      xv[j] = ld_dep(x + base + i);
      rv[j] = ld_dep(residual + base + i);
      wv[j] = w ? __ldg(w + i) : uint16_t(0x3F80);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint64_t i = i0 + j * 256;
      if (i >= k) continue;
      const float n = bf16_round(__fmul_rn(__fmul_rn(to_float(xv[j]), inv), bf16_bits_to_float(wv[j])));
      if (normalized) normalized[base + i] = n;
      float v = bf16_round(__fadd_rn(n, to_float(rv[j])));
      if (scalar) v = bf16_round(__fmul_rn(v, layer_scale));
      store_scalar(out, base + i, v);
    }
  }
}

__device__ __forceinline__ float norm_weight(const uint16_t* w, uint64_t i) {
  return w ? bf16_bits_to_float(__ldg(w + i)) : 1.0f;
}

template <typename In, bool kRcp, bool kInterleaved, bool kShort>
__global__ void __launch_bounds__(256)
rmsnorm_nvfp4_quantize_kernel(const In* x, const uint16_t* __restrict__ w, uint8_t* packed, uint8_t* scales,
                              uint32_t rows, uint64_t k, float eps, float g, uint32_t c_pad) {
  __shared__ float red[256];
  __shared__ __align__(16) float xs[kShort ? kShortRow : 4];
  pdl_trigger();
  const uint64_t r = blockIdx.x;
  const uint32_t c_real = static_cast<uint32_t>(k / 16);
  const bool pad_row = r >= rows;   // interleaved layout only: rows up to a multiple of 128 get zero scales
  constexpr bool short_row = kShort;
  const In* row = x + r * k;
  float inv = 0.0f;
  uint16_t wv[16];
  if (short_row && !pad_row) load_norm_weights(w, threadIdx.x, static_cast<uint32_t>(k), wv);
  pdl_wait();
  if (!pad_row) inv = short_row ? stage_short_row(row, static_cast<uint32_t>(k), eps, xs, red) : rmsnorm_inverse(row, k, eps, red);
  for (uint32_t c0 = 0; c0 < c_pad; c0 += 256) {
    const uint32_t c = c0 + threadIdx.x;
    uint8_t sb = 0;
    if (c < c_real && !pad_row) {
      float v[16];
      if (short_row) {   // one trip: c = threadIdx.x
        normalise_staged(xs, c, wv, inv, v);
      } else {
        load16(row + static_cast<uint64_t>(c) * 16, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = bf16_round(__fmul_rn(__fmul_rn(v[i], inv), norm_weight(w, c * 16ull + i)));
      }
      uint32_t lo, hi;
      quantize_block16<kRcp>(v, g, lo, hi, sb);
      *reinterpret_cast<uint2*>(packed + r * (k / 2) + c * 8ull) = make_uint2(lo, hi);
    }
    const uint32_t word = quad_scale_word(sb);
    if (c >= c_pad) continue;
    if constexpr (kInterleaved) {
      if ((c & 3) == 0) *reinterpret_cast<uint32_t*>(scales + interleaved_scale_offset(r, c, c_pad)) = word;
    } else if (c_real % 4 == 0) {
      if ((c & 3) == 0) *reinterpret_cast<uint32_t*>(scales + r * c_real + c) = word;
    } else if (c < c_real) {
      scales[r * c_real + c] = sb;
    }
  }
}

// FP8 per-token quantizer: pass 1 finds amax (max is order independent), pass 2 divides and converts.
// src/numeric/fp8.cpp:41-58, src/cuda/fp8/reference.cu:39-69.  A thread keeps its first two 16-element
// blocks (rows of up to 8,192 elements) between the passes; the rest of a longer row is read again from L2.
template <typename In, bool kNorm, bool kShort>
__global__ void __launch_bounds__(256)
fp8_quantize_kernel(const In* x, const uint16_t* __restrict__ w, uint8_t* out, float* scales, uint64_t k, float eps) {
  __shared__ float red[256];
  __shared__ float red2[8];
  __shared__ __align__(16) float xs[kNorm && kShort ? kShortRow : 4];
  if constexpr (kNorm) pdl_trigger();
  else pdl_trigger_few_rows(gridDim.x);
  const uint64_t r = blockIdx.x;
  const In* row = x + r * k;
  constexpr bool short_row = kNorm && kShort;
  float inv = 1.0f;
  uint16_t wv[16];
  if (short_row) load_norm_weights(w, threadIdx.x, static_cast<uint32_t>(k), wv);
  if (gridDim.x <= kFewRows) prefetch_l2_span(row, k * sizeof(In));
  pdl_wait();
  if constexpr (kNorm) inv = short_row ? stage_short_row(row, static_cast<uint32_t>(k), eps, xs, red) : rmsnorm_inverse(row, k, eps, red);
  const uint32_t blocks = static_cast<uint32_t>(k / 16);
  auto block_values = [&](uint32_t c, float (&v)[16]) {
    if (short_row) {   // c = threadIdx.x: a short row has at most 256 blocks
      normalise_staged(xs, c, wv, inv, v);
      return;
    }
    load16(row + static_cast<uint64_t>(c) * 16, v);
    if constexpr (kNorm) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = bf16_round(__fmul_rn(__fmul_rn(v[i], inv), norm_weight(w, c * 16ull + i)));
    }
  };
  float kept[2][16];
  float amax = 0.0f;
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const uint32_t c = threadIdx.x + b * 256;
    if (c >= blocks) continue;
    block_values(c, kept[b]);
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(kept[b][i]));
  }
  for (uint32_t c = threadIdx.x + 512; c < blocks; c += 256) {
    float v[16];
    block_values(c, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) red2[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red2[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red2[i]);
  const Quotient q = token_quotient(amax);
  if (threadIdx.x == 0) scales[r] = q.scale;
  uint8_t* orow = out + r * k;
  auto convert = [&](auto code) {
    auto emit = [&](uint32_t c, const float (&v)[16]) {
      uint32_t words[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        words[j] = code(make_float2(v[4 * j], v[4 * j + 1])) | (code(make_float2(v[4 * j + 2], v[4 * j + 3])) << 16);
      *reinterpret_cast<uint4*>(orow + static_cast<uint64_t>(c) * 16) = make_uint4(words[0], words[1], words[2], words[3]);
    };
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (threadIdx.x + b * 256 < blocks) emit(threadIdx.x + b * 256, kept[b]);
    for (uint32_t c = threadIdx.x + 512; c < blocks; c += 256) {
      float v[16];
      block_values(c, v);
      emit(c, v);
    }
  };
  if (q.divide) convert([&](float2 v) { return e4m3x2_divided(v.x, v.y, q.scale); });
  else convert([&](float2 v) { return e4m3_of_quotients(v, q); });
}

// Which form a batch of bf16 rows takes: see the comment above the row kernels.
// Two rows per SM is where a warp per row has as many rows in flight as CTAs per row would.
bool warp_rows(const void* x, const void* w, uint64_t rows, uint64_t k) {
  return rows >= static_cast<uint64_t>(sm_count()) * 2 && k % 16 == 0 && k <= 256 * kRowChunks && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(w) & 15) == 0;
}
template <int kMode, bool kRcp>
int32_t launch_row_warp(const char* op, const RowArgs& a, cudaStream_t stream) {
  const uint64_t rows = kMode == kRowNvfp4Interleaved ? a.rows_out : a.rows;
  GEMB_TRY(launch_pdl(op, row_warp_kernel<kMode, kRcp>, dim3(static_cast<unsigned>((rows + kRowWarps - 1) / kRowWarps)),
                      dim3(kRowWarps * 32), 0, stream, a));
  return check_launch(op);
}

__global__ void __launch_bounds__(256)
interleave_scales_kernel(const uint8_t* __restrict__ compact, uint8_t* __restrict__ out,
                         uint64_t rows, uint64_t c_real, uint64_t rows_pad, uint64_t quads) {
  const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= rows_pad * quads) return;
  const uint64_t r = idx / quads, q = idx % quads;
  uint32_t word = 0;
  if (r < rows)
    for (int j = 0; j < 4; ++j)
      if (q * 4 + j < c_real) word |= static_cast<uint32_t>(__ldg(compact + r * c_real + q * 4 + j)) << (8 * j);
  *reinterpret_cast<uint32_t*>(out + interleaved_scale_offset(r, q * 4, quads * 4)) = word;
}

}  // namespace
}  // namespace gemb

using namespace gemb;

extern "C" {

int32_t gemb_nvfp4_quantize(const void* input, int32_t input_dtype, uint8_t* packed, uint8_t* scales,
                            uint64_t tokens, uint64_t k, float g, int32_t layout, int32_t mode,
                            gemb_stream_t stream) {
  const char* op = "gemb_nvfp4_quantize";
  GEMB_TRY(validate_nvfp4_quantize(op, input, packed, scales, input_dtype, tokens, k, g, layout, mode));
  if (input_dtype == GEMB_F32)
    return launch_nvfp4_quantize(op, PlainLoader<float>{static_cast<const float*>(input)}, packed, scales, tokens, k, g, layout, mode, stream);
  return launch_nvfp4_quantize(op, PlainLoader<uint16_t>{static_cast<const uint16_t*>(input)}, packed, scales, tokens, k, g, layout, mode, stream);
}

int32_t gemb_nvfp4_gated_gelu_quantize(const void* gate, const void* up, int32_t input_dtype,
                                       uint8_t* packed, uint8_t* scales, uint64_t tokens, uint64_t k,
                                       float g, int32_t layout, int32_t mode, gemb_stream_t stream) {
  const char* op = "gemb_nvfp4_gated_gelu_quantize";
  GEMB_REQUIRE(up != nullptr && reinterpret_cast<uintptr_t>(up) % 16 == 0, "%s: up must be nonnull and 16-byte aligned", op);
  GEMB_TRY(validate_nvfp4_quantize(op, gate, packed, scales, input_dtype, tokens, k, g, layout, mode));
  if (input_dtype == GEMB_F32)
    return launch_nvfp4_quantize(op, GatedGeluLoader<float>{static_cast<const float*>(gate), static_cast<const float*>(up)}, packed, scales, tokens, k, g, layout, mode, stream);
  return launch_nvfp4_quantize(op, GatedGeluLoader<uint16_t>{static_cast<const uint16_t*>(gate), static_cast<const uint16_t*>(up)}, packed, scales, tokens, k, g, layout, mode, stream);
}

int32_t gemb_nvfp4_rmsnorm_quantize(const void* input, int32_t input_dtype, const uint16_t* weight,
                                    uint8_t* packed, uint8_t* scales, uint64_t tokens, uint64_t k,
                                    float eps, float g, int32_t layout, int32_t mode,
                                    gemb_stream_t stream) {
  const char* op = "gemb_nvfp4_rmsnorm_quantize";
  GEMB_TRY(validate_nvfp4_quantize(op, input, packed, scales, input_dtype, tokens, k, g, layout, mode));
  GEMB_REQUIRE(std::isfinite(eps) && eps >= 0.0f, "%s: epsilon must be finite and nonnegative", op);
  const bool inter = layout == GEMB_SCALES_INTERLEAVED;
  const bool rcp = mode == GEMB_QUANT_RCP_APPROX;
  const uint64_t c_real = k / 16, c_pad = inter ? (c_real + 3) / 4 * 4 : c_real;
  const uint64_t rows_out = inter ? (tokens + 127) / 128 * 128 : tokens;
  if (input_dtype == GEMB_BF16 && warp_rows(input, weight, tokens, k)) {
    RowArgs a{};
    a.x = input;
    a.w = weight;
    a.out8 = packed;
    a.scales = scales;
    a.rows = tokens;
    a.k = k;
    a.eps = eps;
    a.g = g;
    a.rows_out = static_cast<uint32_t>(rows_out);
    if (inter) return rcp ? launch_row_warp<kRowNvfp4Interleaved, true>(op, a, stream) : launch_row_warp<kRowNvfp4Interleaved, false>(op, a, stream);
    return rcp ? launch_row_warp<kRowNvfp4Compact, true>(op, a, stream) : launch_row_warp<kRowNvfp4Compact, false>(op, a, stream);
  }
  auto launch = [&](auto* x) -> int32_t {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(x)>>;
    auto kern = inter ? (rcp ? rmsnorm_nvfp4_quantize_kernel<T, true, true, false> : rmsnorm_nvfp4_quantize_kernel<T, false, true, false>)
                      : (rcp ? rmsnorm_nvfp4_quantize_kernel<T, true, false, false> : rmsnorm_nvfp4_quantize_kernel<T, false, false, false>);
    if (short_rows(rows_out, k))   // the interleaved layout pads to 128 rows: never
      kern = rcp ? rmsnorm_nvfp4_quantize_kernel<T, true, false, true> : rmsnorm_nvfp4_quantize_kernel<T, false, false, true>;
    GEMB_TRY(launch_pdl_split(op, rows_out <= kFewRows, kern, dim3(static_cast<unsigned>(rows_out)), dim3(256), 0, stream, x, weight, packed, scales,
                              static_cast<uint32_t>(tokens), k, eps, g, static_cast<uint32_t>(c_pad)));
    return check_launch(op);
  };
  return input_dtype == GEMB_F32 ? launch(static_cast<const float*>(input)) : launch(static_cast<const uint16_t*>(input));
}

int32_t gemb_nvfp4_interleave_scales(const uint8_t* compact, uint8_t* interleaved, uint64_t rows,
                                     uint64_t k, gemb_stream_t stream) {
  const char* op = "gemb_nvfp4_interleave_scales";
  GEMB_REQUIRE(compact && interleaved, "%s: pointers must be nonnull", op);
  GEMB_REQUIRE(rows > 0 && k > 0 && k % 16 == 0, "%s: geometry must be nonzero with K a multiple of 16", op);
  GEMB_REQUIRE(reinterpret_cast<uintptr_t>(interleaved) % 4 == 0, "%s: output must be 4-byte aligned", op);
  GEMB_ENTER(op);
  const uint64_t rows_pad = (rows + 127) / 128 * 128, quads = (k / 16 + 3) / 4;
  const unsigned grid = static_cast<unsigned>((rows_pad * quads + 255) / 256);
  interleave_scales_kernel<<<grid, 256, 0, stream>>>(compact, interleaved, rows, k / 16, rows_pad, quads);
  return check_launch(op);
}

static int32_t validate_fp8_quantize(const char* op, const void* in, const void* out, const void* scales,
                                     int32_t dtype, uint64_t tokens, uint64_t k) {
  GEMB_REQUIRE(in && out && scales, "%s: pointers must be nonnull", op);
  GEMB_REQUIRE(dtype == GEMB_F32 || dtype == GEMB_BF16, "%s: input dtype must be GEMB_F32 or GEMB_BF16", op);
  GEMB_REQUIRE(tokens > 0 && k > 0, "%s: token activation must be nonempty", op);
  GEMB_REQUIRE(tokens <= (1ull << 31) - 1 && k <= (1ull << 31), "%s: extent too large", op);
  GEMB_REQUIRE(k % 16 == 0, "%s: elements per token must be a multiple of 16", op);
  GEMB_REQUIRE(reinterpret_cast<uintptr_t>(in) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0,
               "%s: input and output must be 16-byte aligned", op);
  return require_sm100(op);
}

}  // extern "C"
namespace {
template <bool kNorm>
int32_t launch_fp8_rows(const char* op, const void* input, int32_t input_dtype, const uint16_t* weight, uint8_t* out,
                        float* scales, uint64_t tokens, uint64_t k, float eps, cudaStream_t stream) {
  if (input_dtype == GEMB_BF16 && warp_rows(input, weight, tokens, k)) {
    RowArgs a{};
    a.x = input;
    a.w = weight;
    a.out8 = out;
    a.scales = scales;
    a.rows = tokens;
    a.k = k;
    a.eps = eps;
    return launch_row_warp<kNorm ? kRowFp8Norm : kRowFp8, false>(op, a, stream);
  }
  const dim3 grid(static_cast<unsigned>(tokens));
  auto launch = [&](auto* x) -> int32_t {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(x)>>;
    auto kern = kNorm && short_rows(tokens, k) ? fp8_quantize_kernel<T, kNorm, kNorm> : fp8_quantize_kernel<T, kNorm, false>;
    return launch_pdl_split(op, tokens <= kFewRows, kern, grid, dim3(256), 0, stream, x, weight, out, scales, k, eps);
  };
  GEMB_TRY(input_dtype == GEMB_F32 ? launch(static_cast<const float*>(input)) : launch(static_cast<const uint16_t*>(input)));
  return check_launch(op);
}
}  // namespace
extern "C" {

int32_t gemb_fp8_quantize(const void* input, int32_t input_dtype, uint8_t* out, float* scales,
                          uint64_t tokens, uint64_t k, gemb_stream_t stream) {
  const char* op = "gemb_fp8_quantize";
  GEMB_TRY(validate_fp8_quantize(op, input, out, scales, input_dtype, tokens, k));
  if (input_dtype == GEMB_BF16 && tokens <= 16 && k <= 16384)   // decode batches: latency-optimised kernel
    return launch_fp8_quantize_decode(op, static_cast<const uint16_t*>(input), out, scales, tokens, k, stream);
  return launch_fp8_rows<false>(op, input, input_dtype, nullptr, out, scales, tokens, k, 0.0f, stream);
}

int32_t gemb_fp8_rmsnorm_quantize(const void* input, int32_t input_dtype, const uint16_t* weight,
                                  uint8_t* out, float* scales, uint64_t tokens, uint64_t k, float eps,
                                  gemb_stream_t stream) {
  const char* op = "gemb_fp8_rmsnorm_quantize";
  GEMB_TRY(validate_fp8_quantize(op, input, out, scales, input_dtype, tokens, k));
  GEMB_REQUIRE(std::isfinite(eps) && eps >= 0.0f, "%s: epsilon must be finite and nonnegative", op);
  return launch_fp8_rows<true>(op, input, input_dtype, weight, out, scales, tokens, k, eps, stream);
}

int32_t gemb_rmsnorm_residual(const void* input, int32_t input_dtype, const uint16_t* weight_bf16, const void* residual,
                              float* normalized_output, void* output, int32_t residual_output_dtype, uint64_t vectors,
                              uint64_t width, float epsilon, const uint16_t* scalar_bf16, gemb_stream_t stream) {
  const char* op = "gemb_rmsnorm_residual";
  GEMB_REQUIRE(input && residual && output, "%s: input, residual and output must be nonnull", op);
  GEMB_REQUIRE((input_dtype == GEMB_F32 || input_dtype == GEMB_BF16) &&
                   (residual_output_dtype == GEMB_F32 || residual_output_dtype == GEMB_BF16), "%s: unknown dtype", op);
  GEMB_REQUIRE(vectors > 0 && vectors < (1ull << 31) && width > 0 && width < (1ull << 31), "%s: bad geometry", op);
  GEMB_REQUIRE(positive_finite(epsilon), "%s: epsilon must be positive and finite", op);
  GEMB_REQUIRE(residual_output_dtype == GEMB_F32 || (input_dtype == GEMB_BF16 && normalized_output == nullptr),
               "%s: bf16 residual and output go with a bf16 input and no separate normalised output", op);
  GEMB_ENTER(op);
  const bool bf16_out = residual_output_dtype == GEMB_BF16;
  auto aligned16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (bf16_out && warp_rows(input, weight_bf16, vectors, width) && aligned16(residual) && aligned16(output)) {
    RowArgs a{};
    a.x = input;
    a.w = weight_bf16;
    a.residual = residual;
    a.out = output;
    a.scalar = scalar_bf16;
    a.rows = vectors;
    a.k = width;
    a.eps = epsilon;
    return launch_row_warp<kRowResidual, false>(op, a, stream);
  }
  const dim3 grid(static_cast<unsigned>(vectors));
  auto launch = [&](auto* x, auto* res, auto* o) -> int32_t {
    using In = std::remove_const_t<std::remove_pointer_t<decltype(x)>>;
    using Res = std::remove_const_t<std::remove_pointer_t<decltype(res)>>;
    using Out = std::remove_pointer_t<decltype(o)>;
    auto kern = short_rows(vectors, width) ? rmsnorm_residual_kernel<In, Res, Out, true> : rmsnorm_residual_kernel<In, Res, Out, false>;
    return launch_pdl_split(op, vectors <= kFewRows, kern, grid, dim3(256), 0, stream, x, weight_bf16, res, normalized_output, o, width, epsilon, scalar_bf16);
  };
  const auto* xb = static_cast<const uint16_t*>(input);
  if (bf16_out)
    GEMB_TRY(launch(xb, static_cast<const uint16_t*>(residual), static_cast<uint16_t*>(output)));
  else if (input_dtype == GEMB_BF16)
    GEMB_TRY(launch(xb, static_cast<const float*>(residual), static_cast<float*>(output)));
  else
    GEMB_TRY(launch(static_cast<const float*>(input), static_cast<const float*>(residual), static_cast<float*>(output)));
  return check_launch(op);
}

}  // extern "C"
