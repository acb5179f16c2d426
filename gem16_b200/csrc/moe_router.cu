// Router logits: logits[t][e] = fma(x[t][H-1], w[e][H-1], ... fma(x[t][0], w[e][0], bias[e])), one fp32 fma per k in
// ascending k (docs/plans/gemma4-26b/specs/MOE_ROUTER_SPEC.md:3-13,27-38).  The order is the contract: it rules
// out tensor cores and splitting K, so the floor is T x E x H fma on the FMA pipe (128 per clock and SM) and, for
// few tokens, the length of one chain (H x 4 clocks).
#include <algorithm>

#include "common.cuh"

namespace gemb {

// Benchmark hook (GEMB_TUNE_ROUTER_TILE): 0 = automatic, otherwise one of the shapes below.  All give the same bits.
int g_router_tile = 0;

namespace {

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

// ---------------------------------------------------------------------------------------------
// CTA = four warps = 4 kTok tokens x 32 kExp experts: a warp owns kTok tokens, a lane the experts lane + 32 j, so a
// thread carries kTok x kExp independent chains.  What bounds it, per k and SM: kTok kExp clocks of fma, 4 kExp + 2 kTok
// clocks of shared-memory reads (a read returns 128 bytes per clock, broadcast or not; that, 40 clocks
// against 28 of fma per 14 x 4 outputs of a thread, bound the former kernel, which read fp32 tokens), and four clocks of fma latency.
// So the activations stay bf16 in shared memory (one read brings four k of a token) and are widened in
// registers, the weights keep the order memory has them in (rows padded by four words: the lanes' 16-byte reads
// along k are conflict free), and nothing is transposed.
//
// Tiles of 128 / kExp k run through a ring of four buffers by cp.async; one barrier per tile, taken while the tile's
// last operands are in registers, so that neither it nor a shared-memory read is waited for: the
// operands of the next step are always requested before the current step is computed.  2,816 x 128, us before -> now:
// 64 tokens 22.6 -> 14, 256: 29 -> 17, 512: 41 -> 26, 1,024: 53 -> 36, 2,048: 74 -> 57, 3,001: 112 -> 77,
// 6,000: 164 -> 131.  (Loops of two steps instead of the whole tile unrolled: 20-50 % slower; scalar fma
// outgrows the instruction cache with ten and more tokens per warp.)
// ---------------------------------------------------------------------------------------------
constexpr int kRtWarps = 4, kRtThreads = kRtWarps * 32, kRtDepth = 4, kRtSteps = 8;

template <int kTok, int kExp>
struct RouterShape {
  static constexpr int kK = 128 / kExp;            // k per tile
  static constexpr int kStepK = kK / kRtSteps;     // k per step: 16, 8 or 4
  static constexpr int kG = kStepK / 4;            // groups of four k per step
  static constexpr int kTokens = kRtWarps * kTok, kExperts = 32 * kExp;
  struct Smem {
    float w[kRtDepth][kExperts][kK + 4];
    uint16_t x[kRtDepth][kTokens][kK];
  };
};

// The operands of 4 kG consecutive k.
template <int kTok, int kExp, int kG>
struct RouterOps {
  float4 w[kG][kExp];
  uint2 x[kG][kTok];
};

template <int kTok, int kExp, int kG, typename S>
__device__ __forceinline__ void router_load(RouterOps<kTok, kExp, kG>& o, const typename S::Smem& sm, uint32_t buf, int k, int warp, int lane) {
#pragma unroll
  for (int g = 0; g < kG; ++g) {
#pragma unroll
    for (int j = 0; j < kExp; ++j) o.w[g][j] = *reinterpret_cast<const float4*>(&sm.w[buf][lane + 32 * j][k + 4 * g]);
#pragma unroll
    for (int i = 0; i < kTok; ++i) o.x[g][i] = *reinterpret_cast<const uint2*>(&sm.x[buf][warp * kTok + i][k + 4 * g]);
  }
}

// Two tokens share an instruction: the packed fp32 fma is one IEEE fma per half.
template <int kTok, int kExp, int kG>
__device__ __forceinline__ void router_compute(float2 (&acc)[(kTok + 1) / 2][kExp], const RouterOps<kTok, kExp, kG>& o) {
#pragma unroll
  for (int g = 0; g < kG; ++g)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float wq[kExp], xq[kTok];
#pragma unroll
      for (int j = 0; j < kExp; ++j) wq[j] = q == 0 ? o.w[g][j].x : q == 1 ? o.w[g][j].y : q == 2 ? o.w[g][j].z : o.w[g][j].w;
#pragma unroll
      for (int i = 0; i < kTok; ++i) {
        const uint32_t two = q < 2 ? o.x[g][i].x : o.x[g][i].y;
        xq[i] = __uint_as_float((q & 1) ? (two & 0xFFFF0000u) : (two << 16));
      }
      if constexpr (kTok == 1) {
#pragma unroll
        for (int j = 0; j < kExp; ++j) acc[0][j].x = fmaf(xq[0], wq[j], acc[0][j].x);
      } else {
#pragma unroll
        for (int j = 0; j < kExp; ++j) {
          const float2 wp = make_float2(wq[j], wq[j]);
#pragma unroll
          for (int p = 0; p < kTok / 2; ++p) acc[p][j] = __ffma2_rn(make_float2(xq[2 * p], xq[2 * p + 1]), wp, acc[p][j]);
        }
      }
    }
}

template <int kTok, int kExp>
__global__ void __launch_bounds__(kRtThreads, kTok * kExp >= 24 ? 2 : 3)
router_logits_kernel(const uint16_t* x, const float* __restrict__ w, const float* __restrict__ bias, float* logits,
                     uint32_t tokens, uint32_t hidden, uint32_t experts, bool x_wide) {
  using S = RouterShape<kTok, kExp>;
  constexpr int kK = S::kK, kG = S::kG;
  static_assert(kTok == 1 || kTok % 2 == 0, "tokens go in pairs");
  extern __shared__ __align__(16) uint8_t router_smem[];
  auto& sm = *reinterpret_cast<typename S::Smem*>(router_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tok0 = blockIdx.x * S::kTokens, exp0 = blockIdx.y * S::kExperts;
  const uint32_t tiles = (hidden + kK - 1) / kK, full = hidden / kK;
  pdl_trigger();
  pdl_wait();
  // A weight tile is kExperts rows of kK / 4 16-byte pieces (1,024 in all, eight per thread), an activation tile
  // kTokens rows of kK / 8 16-byte pieces (or twice as many halves where rows are only 8-byte aligned).
  constexpr int kWp = kK / 4, kXp = kK / 8;
  const uint32_t wrow = threadIdx.x / kWp, wcol = threadIdx.x % kWp * 4;
  auto issue = [&](uint32_t t) {
    if (t < tiles) {
      const uint32_t k0 = t * kK, buf = t % kRtDepth;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t row = wrow + i * (kRtThreads / kWp);
        const bool ok = k0 + wcol < hidden && exp0 + row < experts;
        cp_async_16(&sm.w[buf][row][wcol], w + static_cast<uint64_t>(ok ? exp0 + row : 0) * hidden + (ok ? k0 + wcol : 0), ok);
      }
      if (x_wide) {
#pragma unroll
        for (int i = 0; i < (S::kTokens * kXp + kRtThreads - 1) / kRtThreads; ++i) {
          const uint32_t idx = threadIdx.x + i * kRtThreads, row = idx / kXp, col = idx % kXp * 8;
          if (row >= static_cast<uint32_t>(S::kTokens)) break;
          const bool ok = k0 + col < hidden && tok0 + row < tokens;
          cp_async_16(&sm.x[buf][row][col], x + static_cast<uint64_t>(ok ? tok0 + row : 0) * hidden + (ok ? k0 + col : 0), ok);
        }
      } else {
#pragma unroll 1
        for (uint32_t idx = threadIdx.x; idx < S::kTokens * kXp * 2u; idx += kRtThreads) {
          const uint32_t row = idx / (kXp * 2), col = idx % (kXp * 2) * 4;
          const bool ok = k0 + col < hidden && tok0 + row < tokens;
          cp_async_8(&sm.x[buf][row][col], x + static_cast<uint64_t>(ok ? tok0 + row : 0) * hidden + (ok ? k0 + col : 0), ok);
        }
      }
    }
    cp_async_commit();   // one group per call, empty past the last tile, so the counting stays uniform
  };
  float2 acc[(kTok + 1) / 2][kExp];
#pragma unroll
  for (int j = 0; j < kExp; ++j) {
    const uint32_t e = exp0 + lane + 32 * j;
    const float b = (bias != nullptr && e < experts) ? __ldg(bias + e) : 0.0f;
#pragma unroll
    for (int p = 0; p < (kTok + 1) / 2; ++p) acc[p][j] = make_float2(b, b);
  }
#pragma unroll
  for (int t = 0; t < kRtDepth; ++t) issue(t);
  cp_async_wait<kRtDepth - 1>();
  __syncthreads();
  RouterOps<kTok, kExp, kG> ops[2];
  router_load<kTok, kExp, kG, S>(ops[0], sm, 0, 0, warp, lane);
  for (uint32_t t = 0; t < full; ++t) {
    const uint32_t buf = t % kRtDepth;
#pragma unroll
    for (int s = 0; s < kRtSteps; ++s) {
      if (s + 1 < kRtSteps) {
        router_load<kTok, kExp, kG, S>(ops[(s + 1) & 1], sm, buf, (s + 1) * S::kStepK, warp, lane);
      } else {
        cp_async_wait<kRtDepth - 2>();   // tile t + 1 has landed (this thread's pieces)
        __syncthreads();                 // everyone's; and everyone has read all of tile t
        issue(t + kRtDepth);             // into the buffer of tile t
        router_load<kTok, kExp, kG, S>(ops[0], sm, (t + 1) % kRtDepth, 0, warp, lane);   // past the last tile: old bytes, not used
      }
      router_compute<kTok, kExp, kG>(acc, ops[s & 1]);
    }
  }
  if (full < tiles) {   // the rest of K, a multiple of four: its tile has landed
    RouterOps<kTok, kExp, 1> o;
#pragma unroll 1
    for (uint32_t k = 0; k < hidden - full * kK; k += 4) {
      router_load<kTok, kExp, 1, S>(o, sm, full % kRtDepth, static_cast<int>(k), warp, lane);
      router_compute<kTok, kExp, 1>(acc, o);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < kTok; ++i) {
    const uint32_t t = tok0 + warp * kTok + i;
    if (t >= tokens) continue;
#pragma unroll
    for (int j = 0; j < kExp; ++j) {
      const uint32_t e = exp0 + lane + 32 * j;
      if (e < experts) logits[static_cast<uint64_t>(t) * experts + e] = (i & 1) ? acc[i / 2][j].y : acc[i / 2][j].x;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The largest batches: CTA = 64 or 56 tokens x 128 experts, thread = 16 or 14 tokens x 4 experts, fp32 tiles of 32 k
// transposed on the way into shared memory, the next tile's global loads in registers.  56 tokens even out
// batches that 64-token CTAs would spread unevenly over the SMs.  Slower than the kernel above while an SM
// has one CTA at most (its loads are then not covered), 15 % faster with two: 16,384 x 2,816 x 128 in 234 us
// (90 of 128 fma per clock and SM) against 274 us, which pays there for widening the activations.  Shared tiles are
// stored k-major with an xor swizzle of the column (multiples of 4 / 8 keep each thread's float4 groups
// intact) so that both the transposing stores and the float4 loads are bank-conflict free.
// ---------------------------------------------------------------------------------------------
constexpr int kRwExp = 128, kRwK = 32;

template <int kTok>
__global__ void __launch_bounds__(kRtThreads, 3)
router_logits_wide_kernel(const uint16_t* __restrict__ x, const float* __restrict__ w,
                     const float* __restrict__ bias, float* __restrict__ logits, uint32_t tokens,
                     uint32_t hidden, uint32_t experts) {
  constexpr int kPerThread = kTok / 4;  // tokens per thread: 16 or 14
  // A warp's tokens occupy a slot of kSlot columns of the shared tile (kSlot = kPerThread rounded up to a
  // multiple of four, so that the float4 reads stay aligned: 16 columns for the 14 tokens of the 56-token tile).
  constexpr int kSlot = (kPerThread + 3) / 4 * 4;
  constexpr int kXCols = 4 * kSlot;
  constexpr int kXLoads = (kTok + 31) / 32;   // staged 16-byte pieces of the token tile per thread
  __shared__ __align__(16) float xs[kRwK][kXCols];
  __shared__ __align__(16) float ws[kRwK][kRwExp];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // experts tx*4.., tokens ty*kPerThread..
  const uint32_t tok0 = blockIdx.x * kTok, exp0 = blockIdx.y * kRwExp;
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
  for (uint32_t k0 = 0; k0 < hidden; k0 += kRwK) {
    store_tile();
    __syncthreads();
    if (k0 + kRwK < hidden) load_tile(k0 + kRwK);
    const uint32_t kmax = min(static_cast<uint32_t>(kRwK), hidden - k0);
    // One k: four weights, kPerThread activations, kPerThread x 4 fma, two tokens to an instruction: every
    // chain keeps its order and rounding while the issue slots carry half the instructions.
    auto step = [&](uint32_t k) {
      const float4 wv4 = *reinterpret_cast<const float4*>(&ws[k][(tx * 4) ^ (4 * (k >> 2))]);
      const float wv[4] = {wv4.x, wv4.y, wv4.z, wv4.w};
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
    };
    if (kmax == kRwK) {
#pragma unroll
      for (uint32_t k = 0; k < kRwK; ++k) step(k);
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

struct RouterArgs {
  const uint16_t* x;
  const float* w;
  const float* bias;
  float* logits;
  uint32_t tokens, hidden, experts;
};

template <int kTok, int kExp>
int32_t launch_router(const char* op, const RouterArgs& a, cudaStream_t stream) {
  using S = RouterShape<kTok, kExp>;
  auto kern = router_logits_kernel<kTok, kExp>;
  GEMB_TRY((allow_full_smem<router_logits_kernel<kTok, kExp>>(op)));
  const bool x_wide = a.hidden % 8 == 0 && reinterpret_cast<uintptr_t>(a.x) % 16 == 0;
  // Not a dependent launch: CTAs placed while the kernel before this one still fills SMs end up two on one SM and none on
  // another (2,048 tokens: 57 us this way, 81 us behind a kernel that triggers early).
  kern<<<dim3((a.tokens + S::kTokens - 1) / S::kTokens, (a.experts + S::kExperts - 1) / S::kExperts), kRtThreads, sizeof(typename S::Smem),
         stream>>>(a.x, a.w, a.bias, a.logits, a.tokens, a.hidden, a.experts, x_wide);
  return check_launch(op);
}
template <int kTok>
int32_t launch_router_wide(const char* op, const RouterArgs& a, cudaStream_t stream) {
  router_logits_wide_kernel<kTok><<<dim3((a.tokens + kTok - 1) / kTok, (a.experts + kRwExp - 1) / kRwExp), kRtThreads, 0, stream>>>(
      a.x, a.w, a.bias, a.logits, a.tokens, a.hidden, a.experts);
  return check_launch(op);
}

// Tokens and experts per CTA, and the measured time (us, 2,816 k) of one CTA per SM and of each further one: the
// shapes that are the fastest for some batch of 128 experts.  Only ratios matter to the choice, and both numbers grow with k but for a
// few microseconds of the first.  Checked against every shape for 64 / 128 / 256 experts, rows of 512 to 6,144 and 15 batches of 1 to
// 12,000 tokens: the choice is within 8 % of the fastest wherever a call takes 10 us or more (within 1.5 us below).
struct RouterShapeCost {
  uint32_t tokens, experts, first, more;
  int32_t (*launch)(const char*, const RouterArgs&, cudaStream_t);
};
constexpr RouterShapeCost kRouterShapes[] = {
    {4, 32, 14, 10, launch_router<1, 1>},      {8, 32, 16, 11, launch_router<2, 1>},      {8, 64, 26, 17, launch_router<2, 2>},
    {16, 64, 35, 27, launch_router<4, 2>},     {32, 64, 57, 46, launch_router<8, 2>},     {24, 128, 77, 64, launch_router<6, 4>},
    {32, 128, 96, 77, launch_router<8, 4>},    {40, 128, 113, 95, launch_router<10, 4>},  {48, 128, 131, 110, launch_router<12, 4>},
    {56, 128, 135, 98, launch_router_wide<56>}, {64, 128, 136, 110, launch_router_wide<64>},
};

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
  const RouterArgs a{x_bf16, router_weight, bias, logits, static_cast<uint32_t>(tokens), static_cast<uint32_t>(hidden), static_cast<uint32_t>(experts)};
  // The shape with the shortest time on the SM that gets the most CTAs.
  const uint64_t sms = static_cast<uint64_t>(sm_count());
  const RouterShapeCost* pick = kRouterShapes;
  uint64_t best = ~0ull;
  for (const RouterShapeCost& c : kRouterShapes) {
    const uint64_t per_sm = ((tokens + c.tokens - 1) / c.tokens * ((experts + c.experts - 1) / c.experts) + sms - 1) / sms;
    const uint64_t cost = c.first + (per_sm - 1) * c.more;
    if (cost < best) {
      best = cost;
      pick = &c;
    }
  }
  if (g_router_tile != 0)   // the n-th shape, or the first one with that many tokens
    for (const RouterShapeCost& c : kRouterShapes)
      if (g_router_tile <= 4 ? &c - kRouterShapes == g_router_tile - 1 : static_cast<int>(c.tokens) == g_router_tile) {
        pick = &c;
        break;
      }
  return pick->launch(op, a, stream);
}
