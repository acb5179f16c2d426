// Router logits: logits[t][e] = fma(x[t][H-1], w[e][H-1], ... fma(x[t][0], w[e][0], bias[e])), one fp32 fma per k in
// ascending k (docs/plans/gemma4-26b/specs/MOE_ROUTER_SPEC.md:3-13,27-38).
#include <algorithm>
#include <atomic>

#include "common.cuh"

namespace gemb {

// Benchmark hook (GEMB_TUNE_ROUTER_TILE): 0 = automatic, 1 = expert-per-thread kernels wherever they
// apply, 8 / 16 / 32 = the tiled kernel with that many tokens per CTA.  All give the same bits.
int g_router_tile = 0;

namespace {

// ---------------------------------------------------------------------------------------------
// Router logits: logits[t][e] = fma(x[t][H-1], w[e][H-1], ... fma(x[t][0], w[e][0], bias[e])),
// one fp32 fma per k in ascending k (the order is the contract; it rules out tensor cores and
// K-splitting).  CTA = 32 tokens x 128 experts, 128 threads, thread = 8 tokens x 4 experts
// (32 independent fma chains).  K is walked in shared-memory tiles of 32; the next tile's global
// loads are issued into registers before the current tile is consumed.
// ---------------------------------------------------------------------------------------------
constexpr int kRtExp = 128, kRtK = 32, kRtThreads = 128;

// kTok = tokens per CTA (64, 56 or 32 for prefill batches -- 64 halves the weight reads from shared memory per
// fma, at 64 accumulators per thread; 56 is the same with 14 tokens per thread, for batches that 64-token
// CTAs would spread unevenly over the SMs -- 8 for decode batches so that a few dozen tokens
// still spread over many SMs).  Shared tiles are stored k-major with an xor swizzle of the column
// (multiples of 4 / 8 keep each thread's float4 groups intact) so that both the transposing
// stores and the float4 loads are bank-conflict free.
template <int kTok>
__global__ void __launch_bounds__(kRtThreads, kTok >= 56 ? 3 : 4)
router_logits_kernel(const uint16_t* __restrict__ x, const float* __restrict__ w,
                     const float* __restrict__ bias, float* __restrict__ logits, uint32_t tokens,
                     uint32_t hidden, uint32_t experts) {
  constexpr int kPerThread = kTok / 4;  // tokens per thread: 16, 14, 8, 4 or 2
  // A warp's tokens occupy a slot of kSlot columns of the shared tile (kSlot = kPerThread rounded up to a
  // multiple of four, so that the float4 reads stay aligned: 16 columns for the 14 tokens of the 56-token tile).
  constexpr int kSlot = kPerThread >= 4 ? (kPerThread + 3) / 4 * 4 : kPerThread;
  constexpr int kXCols = 4 * kSlot > 32 ? 4 * kSlot : 32;
  constexpr int kXLoads = kTok > 32 ? (kTok + 31) / 32 : 1;   // staged 16-byte pieces of the token tile per thread
  __shared__ __align__(16) float xs[kRtK][kXCols];
  __shared__ __align__(16) float ws[kRtK][kRtExp];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // experts tx*4.., tokens ty*kPerThread..
  const uint32_t tok0 = blockIdx.x * kTok, exp0 = blockIdx.y * kRtExp;
  float acc[kPerThread][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t e = exp0 + tx * 4 + j;
    const float b = (bias != nullptr && e < experts) ? __ldg(bias + e) : 0.0f;
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) acc[i][j] = b;
  }
  // Global -> register staging: X tile kTok tokens x 32 k bf16 = one uint4 per thread (token
  // tid/4, k chunk (tid%4)*8); W tile 128 experts x 32 k fp32 = eight float4 per thread
  // (expert tid/8 + 16 i, k chunk (tid%8)*4).
  const int xt = threadIdx.x >> 2, xq = threadIdx.x & 3, xk = xq * 8;
  const int we = threadIdx.x >> 3, wm = threadIdx.x & 7, wk = wm * 4;
  uint4 xr[kXLoads];
  float4 wr[8];
  auto load_tile = [&](uint32_t k0) {
#pragma unroll
    for (int l = 0; l < kXLoads; ++l) {
      xr[l] = make_uint4(0, 0, 0, 0);
      const int tk = xt + 32 * l;   // token of the tile
      if (tk < kTok && tok0 + tk < tokens) {
        const uint16_t* src = x + static_cast<uint64_t>(tok0 + tk) * hidden + k0 + xk;
        if (k0 + xk + 8 <= hidden) {
          if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
            xr[l] = __ldg(reinterpret_cast<const uint4*>(src));
          } else {
            const uint2 a = __ldg(reinterpret_cast<const uint2*>(src)), b2 = __ldg(reinterpret_cast<const uint2*>(src) + 1);
            xr[l] = make_uint4(a.x, a.y, b2.x, b2.y);
          }
        } else if (k0 + xk + 4 <= hidden) {
          const uint2 a = __ldg(reinterpret_cast<const uint2*>(src));
          xr[l] = make_uint4(a.x, a.y, 0, 0);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      wr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      const uint32_t e = exp0 + we + 16 * i;
      if (e < experts && k0 + wk < hidden)
        wr[i] = __ldg(reinterpret_cast<const float4*>(w + static_cast<uint64_t>(e) * hidden + k0 + wk));
    }
  };
  auto store_tile = [&]() {
#pragma unroll
    for (int l = 0; l < kXLoads; ++l) {
      const uint32_t xw[4] = {xr[l].x, xr[l].y, xr[l].z, xr[l].w};
      const int tk = xt + 32 * l;
      if (tk >= kTok) continue;
      const int xcol = ((tk / kPerThread) * kSlot + tk % kPerThread) ^ (8 * xq);  // rows xk..xk+7 all have (k / 8) & 3 == xq
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        xs[xk + 2 * i][xcol] = __uint_as_float(xw[i] << 16);
        xs[xk + 2 * i + 1][xcol] = __uint_as_float(xw[i] & 0xFFFF0000u);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int col = (we + 16 * i) ^ (4 * wm);  // rows wk..wk+3 all have k / 4 == wm
      ws[wk + 0][col] = wr[i].x;
      ws[wk + 1][col] = wr[i].y;
      ws[wk + 2][col] = wr[i].z;
      ws[wk + 3][col] = wr[i].w;
    }
  };
  load_tile(0);
  for (uint32_t k0 = 0; k0 < hidden; k0 += kRtK) {
    store_tile();
    __syncthreads();
    if (k0 + kRtK < hidden) load_tile(k0 + kRtK);
    const uint32_t kmax = min(static_cast<uint32_t>(kRtK), hidden - k0);
    // One k: four weights, kPerThread activations, kPerThread x 4 fma.  With four or eight tokens per
    // thread two tokens share an instruction: the packed fp32 fma is one IEEE fma per half, so every
    // chain keeps its order and rounding while the issue slots carry half the instructions.
    auto step = [&](uint32_t k) {
      const float4 wv4 = *reinterpret_cast<const float4*>(&ws[k][(tx * 4) ^ (4 * (k >> 2))]);
      const float wv[4] = {wv4.x, wv4.y, wv4.z, wv4.w};
      const int col = (ty * kPerThread) ^ (8 * ((k >> 3) & 3));
      if constexpr (kPerThread >= 4) {
        float2 xp[kPerThread / 2];
#pragma unroll
        for (int q = 0; q < kSlot / 4; ++q) {   // the swizzle moves groups of eight columns: a group of four stays whole
          const float4 xa = *reinterpret_cast<const float4*>(&xs[k][(ty * kSlot + 4 * q) ^ (8 * ((k >> 3) & 3))]);
          xp[2 * q] = make_float2(xa.x, xa.y);
          if (2 * q + 1 < kPerThread / 2) xp[2 * q + 1] = make_float2(xa.z, xa.w);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 wp = make_float2(wv[j], wv[j]);
#pragma unroll
          for (int i = 0; i < kPerThread / 2; ++i) {
            const float2 r = __ffma2_rn(xp[i], wp, make_float2(acc[2 * i][j], acc[2 * i + 1][j]));
            acc[2 * i][j] = r.x;
            acc[2 * i + 1][j] = r.y;
          }
        }
      } else {
        const float2 xa = *reinterpret_cast<const float2*>(&xs[k][col]);
        const float xv[2] = {xa.x, xa.y};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
      }
    };
    if (kmax == kRtK) {
#pragma unroll
      for (uint32_t k = 0; k < kRtK; ++k) step(k);
    } else {
#pragma unroll 4
      for (uint32_t k = 0; k < kmax; ++k) step(k);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < kPerThread; ++i) {
    const uint32_t t = tok0 + ty * kPerThread + i;
    if (t >= tokens) continue;
    float* dst = logits + static_cast<uint64_t>(t) * experts + exp0 + tx * 4;
    if (exp0 + tx * 4 + 4 <= experts && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
      *reinterpret_cast<float4*>(dst) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (exp0 + tx * 4 + j < experts) dst[j] = acc[i][j];
    }
  }
}

// Decode-size and small-batch form of the same contract.  With few tokens the tile above leaves
// most SMs idle (one CTA per 8 or 32 tokens, each walking all of K).  Here a thread owns ONE
// expert and kTpt tokens (kTpt independent fma chains), a warp 32 experts, a CTA of two warps
// 2 * kTpt tokens of the same 32 experts.  K is walked in tiles of 128.  The chain over k is
// serial, so a tile's arithmetic (about 600 clocks) is all there is to hide a load behind, and
// an L2 round trip takes longer than that: the CTA's weight tiles (32 experts x 128 k, fetched
// as coalesced 16-byte cp.async pieces) and the tokens' raw bf16 activations therefore run
// through a ring of kRsDepth shared-memory buffers, three tiles ahead of the arithmetic.  Same
// chain, same order: bias, then one fma per k ascending.
constexpr int kRsK = 128, kRsThreads = 64, kRsPad = 4, kRsDepth = 4;

__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* src, bool valid) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  const uint32_t n = valid ? 16u : 0u;   // 0 source bytes: the destination is zero filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_8(void* smem_dst, const void* src, bool valid) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  const uint32_t n = valid ? 8u : 0u;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }

template <int kTpt>
struct RouterSmallSmem {
  static constexpr int kTokCta = 2 * kTpt;
  float ws[kRsDepth][32][kRsK + kRsPad];     // row stride 132 words: float4 reads of one k by 32 rows are conflict free
  uint16_t xraw[kRsDepth][kTokCta][kRsK];    // bf16 as loaded
  float xs[kTokCta][kRsK];                   // the current tile's activations as fp32
};

template <int kTpt>
__global__ void __launch_bounds__(kRsThreads)
router_logits_small_kernel(const uint16_t* __restrict__ x, const float* __restrict__ w,
                           const float* __restrict__ bias, float* __restrict__ logits, uint32_t tokens,
                           uint32_t hidden, uint32_t experts) {
  constexpr int kTokCta = 2 * kTpt;
  extern __shared__ __align__(16) uint8_t router_small_smem[];
  auto& sm = *reinterpret_cast<RouterSmallSmem<kTpt>*>(router_small_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tok0 = blockIdx.x * kTokCta, exp0 = blockIdx.y * 32;
  const uint32_t e = exp0 + lane;
  const bool live = e < experts;
  float acc[kTpt];
  const float b = (bias != nullptr && live) ? __ldg(bias + e) : 0.0f;
#pragma unroll
  for (int i = 0; i < kTpt; ++i) acc[i] = b;
  const uint32_t tiles = (hidden + kRsK - 1) / kRsK;
  // Warp `warp` fetches rows warp*16 .. warp*16+15 of the weight tile (lane = 16-byte piece of the
  // row); the activation tile is kTokCta rows of 32 eight-byte pieces shared out over the CTA.
  auto issue_tile = [&](uint32_t t) {
    if (t < tiles) {
      const uint32_t k0 = t * kRsK, buf = t % kRsDepth;
      const uint32_t kmax = min(static_cast<uint32_t>(kRsK), hidden - k0);   // a multiple of 4
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const uint32_t row = exp0 + warp * 16 + r;
        const bool ok = row < experts && static_cast<uint32_t>(lane) * 4 < kmax;
        const float* src = w + static_cast<uint64_t>(ok ? row : 0) * hidden + (ok ? k0 + lane * 4 : 0);
        cp_async_16(&sm.ws[buf][warp * 16 + r][lane * 4], src, ok);
      }
#pragma unroll
      for (int q = 0; q < kTokCta * 32 / kRsThreads; ++q) {
        const uint32_t idx = threadIdx.x + q * kRsThreads;
        const uint32_t tk = idx / 32, c = (idx % 32) * 4;
        const bool ok = tok0 + tk < tokens && c < kmax;
        const uint16_t* src = x + static_cast<uint64_t>(ok ? tok0 + tk : 0) * hidden + (ok ? k0 + c : 0);
        cp_async_8(&sm.xraw[buf][tk][c], src, ok);
      }
    }
    cp_async_commit();   // one group per call, empty past the last tile, so the counting stays uniform
  };
#pragma unroll
  for (int t = 0; t < kRsDepth - 1; ++t) issue_tile(t);
  for (uint32_t t = 0; t < tiles; ++t) {
    const uint32_t buf = t % kRsDepth;
    const uint32_t groups = min(static_cast<uint32_t>(kRsK), hidden - t * kRsK) / 4;
    cp_async_wait<kRsDepth - 2>();   // this thread's pieces of tile t have landed
    __syncthreads();                 // everyone's have; and tile t-1 has been consumed
    issue_tile(t + kRsDepth - 1);    // refills the buffer tile t-1 used
    for (uint32_t idx = threadIdx.x; idx < kTokCta * (kRsK / 4); idx += kRsThreads) {
      const uint32_t tk = idx / (kRsK / 4), c = (idx % (kRsK / 4)) * 4;
      const uint2 raw = *reinterpret_cast<const uint2*>(&sm.xraw[buf][tk][c]);
      *reinterpret_cast<float4*>(&sm.xs[tk][c]) =
          make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xFFFF0000u),
                      __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xFFFF0000u));
    }
    __syncthreads();
#pragma unroll 8
    for (uint32_t g = 0; g < groups; ++g) {
      const float4 wv = *reinterpret_cast<const float4*>(&sm.ws[buf][lane][g * 4]);
      float4 xv[kTpt];
#pragma unroll
      for (int i = 0; i < kTpt; ++i) xv[i] = *reinterpret_cast<const float4*>(&sm.xs[warp * kTpt + i][g * 4]);
      // k-major: the kTpt chains advance together, so consecutive instructions are independent
      // (a chain's own steps are four clocks apart at best).
#pragma unroll
      for (int i = 0; i < kTpt; ++i) acc[i] = fmaf(xv[i].x, wv.x, acc[i]);
#pragma unroll
      for (int i = 0; i < kTpt; ++i) acc[i] = fmaf(xv[i].y, wv.y, acc[i]);
#pragma unroll
      for (int i = 0; i < kTpt; ++i) acc[i] = fmaf(xv[i].z, wv.z, acc[i]);
#pragma unroll
      for (int i = 0; i < kTpt; ++i) acc[i] = fmaf(xv[i].w, wv.w, acc[i]);
    }
  }
  cp_async_wait<0>();
  if (!live) return;
#pragma unroll
  for (int i = 0; i < kTpt; ++i) {
    const uint32_t t = tok0 + warp * kTpt + i;
    if (t < tokens) logits[static_cast<uint64_t>(t) * experts + e] = acc[i];
  }
}
// The small-batch router kernel's ring needs more than the 48 KB a kernel gets without opting in.
template <int kTpt>
int32_t router_small_configure(const char* op) {
  static std::atomic<bool> configured[64];   // racing first calls both set the (idempotent) attribute
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!configured[dev].load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(router_logits_small_kernel<kTpt>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(RouterSmallSmem<kTpt>)));
    if (e != cudaSuccess) return fail(GEMB_INTERNAL, "%s: %s: %s", op, cudaGetErrorName(e), cudaGetErrorString(e));
    configured[dev].store(true, std::memory_order_release);
  }
  return GEMB_OK;
}
}  // namespace
}  // namespace gemb

using namespace gemb;

extern "C" int32_t gemb_moe_router_logits(const uint16_t* x_bf16, const float* router_weight, const float* bias,
                               float* logits, uint64_t tokens, uint64_t hidden, uint64_t experts,
                               gemb_stream_t stream) {
  const char* op = "gemb_moe_router_logits";
  GEMB_REQUIRE(x_bf16 && router_weight && logits, "%s: pointers must be nonnull", op);
  GEMB_REQUIRE(tokens > 0 && tokens < (1ull << 31) && experts > 0 && experts < (1ull << 20), "%s: bad geometry", op);
  GEMB_REQUIRE(hidden > 0 && hidden % 4 == 0 && hidden < (1ull << 31), "%s: hidden must be a nonzero multiple of 4", op);
  GEMB_REQUIRE(reinterpret_cast<uintptr_t>(x_bf16) % 8 == 0 && reinterpret_cast<uintptr_t>(router_weight) % 16 == 0,
               "%s: activations must be 8-byte and router weights 16-byte aligned", op);
  GEMB_ENTER(op);
  // Up to a thousand tokens: one expert per thread, weight rows streamed from L2 (the tiled kernel
  // would occupy a fraction of the SMs).  Its L2 traffic grows with the token count (one pass over
  // the router weight per 2 * kTpt tokens), so larger batches use the tiled kernel.  Measured on
  // 2,816 x 128: 25 / 31 / 43 / 56 us at 64 / 256 / 512 / 1,024 tokens here, against 64 us for the
  // tiled kernel; at 2,048 tokens 105 us against 72 us for the 16-token tile.
  if ((tokens <= 1024 && g_router_tile == 0) || (tokens <= 2048 && g_router_tile == 1)) {
    if (tokens <= 256) {
      dim3 g(static_cast<unsigned>((tokens + 3) / 4), static_cast<unsigned>((experts + 31) / 32));
      GEMB_TRY(router_small_configure<2>(op));
      router_logits_small_kernel<2><<<g, kRsThreads, sizeof(RouterSmallSmem<2>), stream>>>(x_bf16, router_weight, bias, logits,
                                                                   static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                                   static_cast<uint32_t>(experts));
    } else if (tokens <= 512) {
      dim3 g(static_cast<unsigned>((tokens + 7) / 8), static_cast<unsigned>((experts + 31) / 32));
      GEMB_TRY(router_small_configure<4>(op));
      router_logits_small_kernel<4><<<g, kRsThreads, sizeof(RouterSmallSmem<4>), stream>>>(x_bf16, router_weight, bias, logits,
                                                                   static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                                   static_cast<uint32_t>(experts));
    } else {
      dim3 g(static_cast<unsigned>((tokens + 15) / 16), static_cast<unsigned>((experts + 31) / 32));
      GEMB_TRY(router_small_configure<8>(op));
      router_logits_small_kernel<8><<<g, kRsThreads, sizeof(RouterSmallSmem<8>), stream>>>(x_bf16, router_weight, bias, logits,
                                                                   static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                                   static_cast<uint32_t>(experts));
    }
    return check_launch(op);
  }
  // 8- and 16-token CTAs only while they do not outnumber the SMs; beyond that the larger tiles do more
  // arithmetic per shared-memory load: 32 tokens, and 64 once there is a 64-token CTA for most SMs
  // (measured on 2,816 x 128: 303 / 268 us at 16,384 tokens, 166 / 158 us at 8,192, 114 / 158 us at 4,096).
  const uint64_t expert_tiles = (experts + kRtExp - 1) / kRtExp;
  unsigned tile = 32;
  if ((tokens + 7) / 8 * expert_tiles <= static_cast<uint64_t>(sm_count())) tile = 8;
  else if ((tokens + 15) / 16 * expert_tiles <= static_cast<uint64_t>(sm_count())) tile = 16;
  else if ((tokens + 63) / 64 * expert_tiles * 8 >= static_cast<uint64_t>(sm_count()) * 6) tile = 64;
  // 56-token CTAs where they even out the load: with up to two of the large CTAs per SM, an SM's time goes with
  // the tokens it holds (16,384 tokens: 256 CTAs of 64 leave 40 SMs with one CTA and 108 with two, 293 CTAs
  // of 56 give every SM two).
  if (tile == 64) {
    const uint64_t sms = static_cast<uint64_t>(sm_count());
    const uint64_t c64 = (tokens + 63) / 64 * expert_tiles, c56 = (tokens + 55) / 56 * expert_tiles;
    if ((c56 + sms - 1) / sms * 56 < (c64 + sms - 1) / sms * 64) tile = 56;
  }
  if (g_router_tile == 8 || g_router_tile == 16 || g_router_tile == 32 || g_router_tile == 56 || g_router_tile == 64)
    tile = static_cast<unsigned>(g_router_tile);
  dim3 grid(static_cast<unsigned>((tokens + tile - 1) / tile), static_cast<unsigned>((experts + kRtExp - 1) / kRtExp));
  if (tile == 8)
    router_logits_kernel<8><<<grid, kRtThreads, 0, stream>>>(x_bf16, router_weight, bias, logits,
                                                            static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                            static_cast<uint32_t>(experts));
  else if (tile == 16)
    router_logits_kernel<16><<<grid, kRtThreads, 0, stream>>>(x_bf16, router_weight, bias, logits,
                                                             static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                             static_cast<uint32_t>(experts));
  else if (tile == 56)
    router_logits_kernel<56><<<grid, kRtThreads, 0, stream>>>(x_bf16, router_weight, bias, logits,
                                                             static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                             static_cast<uint32_t>(experts));
  else if (tile == 64)
    router_logits_kernel<64><<<grid, kRtThreads, 0, stream>>>(x_bf16, router_weight, bias, logits,
                                                             static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                             static_cast<uint32_t>(experts));
  else
    router_logits_kernel<32><<<grid, kRtThreads, 0, stream>>>(x_bf16, router_weight, bias, logits,
                                                             static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden),
                                                             static_cast<uint32_t>(experts));
  return check_launch(op);
}
