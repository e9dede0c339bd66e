// Top-k router: MoEGate.forward of moe/all2all_moe.py:60-118, one launch.
//
// Phase A computes f32 logits x . W^T for a tile of tokens into shared memory;
// phase B (one warp per token) applies sigmoid/softmax, the group-limited
// selection and the weight normalisation.  Ties always go to the lower expert
// id, so the output is a pure function of the scores.
//
//   E <= 32  : one warp per token, 128-bit loads of x, shuffle reductions
//              (HBM-bound: x is read once, W stays in L1/L2)
//   E <= 256 : 32-token x E register-tiled f32 GEMM through shared memory
#include "common.cuh"

namespace b200moe {

constexpr int kMaxE = 256;
constexpr int kMaxTopK = 32;

struct RouterParams {
  const float* w;      // [E,H]
  const float* bias;   // [E] or null
  int64_t T, H;
  int E, top_k, n_group, topk_group, scoring, norm;
  float scale;
  int64_t* topk_idx;
  float* topk_weight;
};

// Unsigned image of a float that orders like it (-0 and +0 alike); 0 is below every number's.
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t u = __float_as_uint(v + 0.0f);
  return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}

// Scores of one token's experts from their logits, in place in shared memory, by the calling warp (softmax; sigmoid scores need
// no other expert and are formed where the logits are).
__device__ __forceinline__ void softmax_scores(float* logit, int E) {
  const int lane = threadIdx.x & 31;
  float m = -INFINITY;
#pragma unroll 1
  for (int e = lane; e < E; e += 32) m = fmaxf(m, logit[e]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  float sum = 0.f;
#pragma unroll 1
  for (int e = lane; e < E; e += 32) { const float ex = expf(logit[e] - m); logit[e] = ex; sum += ex; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll 1
  for (int e = lane; e < E; e += 32) logit[e] = __fdiv_rn(logit[e], sum);
}
__device__ __forceinline__ float sigmoid_score(float logit) { return __fdiv_rn(1.f, 1.f + expf(-logit)); }

// Phase B for one token by one warp.  `score` holds the E scores, `sfc` is E floats of scratch (used by the group selection
// only), both in shared memory and private to the warp; J registers per lane cover E experts.
//
// What bounds it: the latency of eight dependent picks for a token, and for few tokens the fetch of this code.  The candidates
// stay in registers and a pick is two redux.sync on integer images of the scores; with the candidates in shared memory, a pick
// was eight loads and ten shuffles and the scan of the groups met itself in one bank.
template <int J>
__device__ void select_token(const RouterParams& p, int64_t t, const float* score, float* sfc) {
  const int lane = threadIdx.x & 31;
  const int E = p.E;
  float s[J];                                            // selection scores
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int e = lane + 32 * j;
    s[j] = e < E ? score[e] + (p.bias ? p.bias[e] : 0.f) : -INFINITY;
  }

  if (p.n_group > 1) {
    // group score = sum of the two largest selection scores of the group, whose members are dealt to `width` lanes; the scan
    // starts at another member in every group, so that lanes of different groups read different banks
#pragma unroll
    for (int j = 0; j < J; ++j) if (lane + 32 * j < E) sfc[lane + 32 * j] = s[j];
    __syncwarp();
    const int gsz = E / p.n_group;
    int width = 32;
    while (width * p.n_group > 32) width >>= 1;
    const int g = lane / width, sub = lane - g * width;
    float a = -INFINITY, b = -INFINITY;
    if (g < p.n_group) {
      const int n = (gsz - sub + width - 1) / width;     // members of this lane: sub, sub + width, ...
      for (int i = 0, k = n > 0 ? g % n : 0; i < n; ++i, k = k + 1 < n ? k + 1 : 0) {
        const float x = sfc[g * gsz + sub + k * width];
        if (x > a) { b = a; a = x; } else if (x > b) { b = x; }
      }
    }
    for (int o = width >> 1; o > 0; o >>= 1) {
      const float oa = __shfl_xor_sync(0xffffffffu, a, o), ob = __shfl_xor_sync(0xffffffffu, b, o);
      b = fmaxf(fminf(a, oa), fmaxf(b, ob));
      a = fmaxf(a, oa);
    }
    const float gs = __shfl_sync(0xffffffffu, a + b, (lane * width) & 31);
    const uint32_t lowest = order_key(-INFINITY);
    uint32_t key = lane < p.n_group ? (gs == gs ? order_key(gs) : lowest) : 0u;
    uint32_t keep = 0;                                   // bit g set = group g survives (n_group <= 32)
    for (int r = 0; r < p.topk_group; ++r) {
      const uint32_t best = __reduce_max_sync(0xffffffffu, key);
      const int i = static_cast<int>(__reduce_min_sync(0xffffffffu, key == best ? static_cast<uint32_t>(lane) : 32u));
      keep |= 1u << i;
      if (lane == i) key = lowest;
    }
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int e = lane + 32 * j;
      if (e < E && !((keep >> (e / gsz)) & 1u)) s[j] = 0.0f;     // masked_fill(~mask, 0.0)
    }
  }

  // top-k over the selection scores; NaN and -inf are no candidates
  uint32_t key[J];
#pragma unroll
  for (int j = 0; j < J; ++j) key[j] = s[j] > -INFINITY ? order_key(s[j]) : 0u;
  float wsum = 0.f;
  float my_w = 0.f; int my_i = 0;   // lane r keeps the r-th pick
  for (int r = 0; r < p.top_k; ++r) {
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < J; ++j) m = max(m, key[j]);
    const uint32_t best = __reduce_max_sync(0xffffffffu, m);
    uint32_t cand = 0xffffffffu;
#pragma unroll
    for (int j = J - 1; j >= 0; --j) if (key[j] == best) cand = static_cast<uint32_t>(lane + 32 * j);
    const int i = best == 0u ? 0 : static_cast<int>(__reduce_min_sync(0xffffffffu, cand));   // ties: the lower id
#pragma unroll
    for (int j = 0; j < J; ++j) if (i == lane + 32 * j) key[j] = 0u;
    const float sc = score[i];
    if (lane == r) { my_w = sc; my_i = i; }
    wsum += sc;
  }
  if (lane < p.top_k) {
    float wv = my_w;
    if (p.top_k > 1 && p.norm) wv = __fdiv_rn(wv, wsum + 1e-20f);
    wv *= p.scale;
    p.topk_idx[t * p.top_k + lane] = my_i;
    p.topk_weight[t * p.top_k + lane] = wv;
  }
}

// The same from logits in shared memory.
template <int J>
__device__ __forceinline__ void select_from_logits(const RouterParams& p, int64_t t, float* logit, float* sfc) {
  if (p.scoring == 1) softmax_scores(logit, p.E);
  else {
#pragma unroll 1
    for (int e = threadIdx.x & 31; e < p.E; e += 32) logit[e] = sigmoid_score(logit[e]);
  }
  __syncwarp();
  select_token<J>(p, t, logit, sfc);
}

// ---- E <= 32: warp per token ------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) router_small_kernel(const T* __restrict__ x, RouterParams p) {
  __shared__ float s_logit[8][32];
  __shared__ float s_sfc[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * 8 + warp;
  if (t >= p.T) return;
  const int E = p.E;
  float acc[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) acc[e] = 0.f;
  const T* xr = x + t * p.H;
  for (int64_t h = lane * 8; h < p.H; h += 256) {
    float xv[8];
    load8(xr + h, xv);
#pragma unroll
    for (int e = 0; e < 32; ++e) {
      if (e < E) {
        float wv[8];
        load8(p.w + e * p.H + h, wv);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[e] = fmaf(xv[k], wv[k], acc[e]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    if (e < E) {
      float v = acc[e];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) s_logit[warp][e] = v;
    }
  }
  __syncwarp();
  select_from_logits<1>(p, t, s_logit[warp], s_sfc[warp]);
}

// ---- E <= 256: 32 tokens x E tile, K chunks of 32 through shared memory -----------
constexpr int kTM = 32;   // tokens per CTA
constexpr int kKC = 32;   // K chunk
constexpr int kLd = kKC + 4;

template <typename T>
__global__ void __launch_bounds__(256) router_tiled_kernel(const T* __restrict__ x, RouterParams p) {
  extern __shared__ __align__(16) float smem[];
  float* xs = smem;                       // [kTM][kLd]
  float* ws = xs + kTM * kLd;             // [kMaxE][kLd]
  float* lg = ws + kMaxE * kLd;           // [kTM][kMaxE] logits, later scores
  float* sf = lg + kTM * kMaxE;           // [8][kMaxE] per-warp selection scratch
  const int tid = threadIdx.x;
  const int tx = tid & 31, ty = tid >> 5;  // ty: 4 tokens each; tx: experts tx + 32 j
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * kTM;
  const int E = p.E;
  float acc[4][8];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[a][b] = 0.f;

  for (int64_t k0 = 0; k0 < p.H; k0 += kKC) {
    // x tile: 32 tokens x 32 k = 128 chunks of 8 -> threads 0..127
    if (tid < 128) {
      const int r = tid >> 2, c = (tid & 3) * 8;
      float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (t0 + r < p.T && k0 + c < p.H) load8(x + (t0 + r) * p.H + k0 + c, v);
      store8(xs + r * kLd + c, v);
    }
    // W tile: E x 32 k = E*4 chunks of 8
    for (int i = tid; i < E * 4; i += 256) {
      const int r = i >> 2, c = (i & 3) * 8;
      float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (k0 + c < p.H) load8(p.w + static_cast<int64_t>(r) * p.H + k0 + c, v);
      store8(ws + r * kLd + c, v);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kKC; kk += 4) {
      float4 xv[4], wv[8];
#pragma unroll
      for (int a = 0; a < 4; ++a) xv[a] = *reinterpret_cast<const float4*>(xs + (ty * 4 + a) * kLd + kk);
#pragma unroll
      for (int b = 0; b < 8; ++b)
        wv[b] = (tx + 32 * b < E) ? *reinterpret_cast<const float4*>(ws + (tx + 32 * b) * kLd + kk)
                                  : make_float4(0, 0, 0, 0);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          acc[a][b] = fmaf(xv[a].x, wv[b].x, acc[a][b]);
          acc[a][b] = fmaf(xv[a].y, wv[b].y, acc[a][b]);
          acc[a][b] = fmaf(xv[a].z, wv[b].z, acc[a][b]);
          acc[a][b] = fmaf(xv[a].w, wv[b].w, acc[a][b]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b)
      if (tx + 32 * b < E) lg[(ty * 4 + a) * kMaxE + tx + 32 * b] = acc[a][b];
  __syncthreads();
  for (int a = 0; a < 4; ++a) {
    const int64_t t = t0 + ty * 4 + a;
    if (t < p.T) select_from_logits<kMaxE / 32>(p, t, lg + (ty * 4 + a) * kMaxE, sf + ty * kMaxE);
    __syncwarp();
  }
}

// ---- logits of few tokens ------------------------------------------------------------------
// logits[t, e] = x[t] . w[e] in f32, w given as its three bf16 parts side by side (hi + mid + lo = w exactly).  Bound by the
// 6 E H bytes of the parts.  A block takes two experts and up to two tokens, four warps an expert, each a quarter of the columns;
// their sums are added in order.
constexpr int kFewTokens = static_cast<int>(kRouterFewTokens);
static_assert((kFewTokens & (kFewTokens - 1)) == 0, "tokens of a block are told apart by a mask");
__global__ void __launch_bounds__(256) router_few_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w3,
                                                         float* __restrict__ logits, int64_t T, int64_t H, int E) {
  __shared__ float part[8][kFewTokens];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e = static_cast<int>(blockIdx.x) * 2 + (warp >> 2);       // E is a multiple of 128
  const int64_t t0 = static_cast<int64_t>(blockIdx.y) * kFewTokens;
  const int tokens = static_cast<int>(min(T - t0, static_cast<int64_t>(kFewTokens)));
  const __nv_bfloat16* w = w3 + static_cast<int64_t>(e) * 3 * H;
  float acc[kFewTokens];
#pragma unroll
  for (int k = 0; k < kFewTokens; ++k) acc[k] = 0.f;
  wait_for_predecessors();
  allow_dependents();
#pragma unroll 2
  for (int64_t h = ((warp & 3) * 32 + lane) * 8; h < H; h += 1024) {  // H is a multiple of 64
    float hi[8], mid[8], lo[8];
    load8(w + h, hi);
    load8(w + H + h, mid);
    load8(w + 2 * H + h, lo);
#pragma unroll
    for (int i = 0; i < 8; ++i) hi[i] = (hi[i] + mid[i]) + lo[i];
#pragma unroll
    for (int k = 0; k < kFewTokens; ++k) {
      if (k >= tokens) break;
      float v[8];
      load8(x + (t0 + k) * H + h, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[k] = fmaf(v[i], hi[i], acc[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < kFewTokens; ++k) {
    if (k >= tokens) break;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (lane == 0) part[warp][k] = acc[k];
  }
  __syncthreads();
  if (threadIdx.x < 2 * kFewTokens) {
    const int k = threadIdx.x & (kFewTokens - 1), g = threadIdx.x / kFewTokens;
    if (k < tokens)
      logits[(t0 + k) * E + static_cast<int64_t>(blockIdx.x) * 2 + g] =
          ((part[g * 4][k] + part[g * 4 + 1][k]) + part[g * 4 + 2][k]) + part[g * 4 + 3][k];
  }
}

int router_logits_few(const void* x_bf16, const void* w3_bf16, float* logits, int64_t T, int64_t H, int E, cudaStream_t st) {
  const dim3 grid(static_cast<unsigned>(E / 2), static_cast<unsigned>((T + kFewTokens - 1) / kFewTokens));
  return launch_dependent("router_logits", router_few_kernel, grid, 256, 0, st, static_cast<const __nv_bfloat16*>(x_bf16),
                          static_cast<const __nv_bfloat16*>(w3_bf16), logits, T, H, E);
}

// ---- selection from precomputed logits (tensor-core path) ----------------------------------
// Eight tokens per block, a warp selects for one; J registers per lane cover E experts.  What bounds it: the latency of the loads
// of the partial sums, so many of them are in flight, and for a token or two the fetch of the code.
//
// Few tokens (they fit side by side in the block's threads; with more than 256 experts, one or two): a thread per expert, short
// code with eight splits in flight.  More tokens: each warp adds its own, J experts a lane, 32 (J 8, 32) or 64 (J 16) loads in
// flight; with the first form for all, 16 splits took eight rounds of 16 loads one after another.  us, 16 splits, first form -> a
// warp each: 256 experts, top-8 of 8 groups: one token 6.1 -> 6.9, two 8.3 -> 6.7, 77 tokens 18 -> 7.6, 4096 35 -> 17, 8192
// 83 -> 36; 384 experts, one token 5.7 -> 6.9, two 7.6 -> 6.8, 4096 72 -> 25; 1024 experts, one token 16 -> 19, three 21 -> 19,
// 4096 132 -> 70.
//
// Registers: 80 for 256 experts, where the compiler takes 64 by itself (one token 6.9 -> 6.1 us, 4096 tokens 15.4 -> 17.2); 48 up to
// 32 experts (eight experts, 4096 tokens: 4.5 us, 5.2 with 80).
constexpr int kSelectTokens = 8;
template <int J>
__global__ void __launch_bounds__(256, J == 1 ? 5 : 1) router_select_kernel(const float* __restrict__ partials,
                                                            int nsplit, int64_t row_stride, RouterParams p) {
  extern __shared__ __align__(16) float smem[];   // [8 tokens][2][E]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * kSelectTokens;
  wait_for_predecessors();
  allow_dependents();
  const int tokens = static_cast<int>(min(p.T - t0, static_cast<int64_t>(kSelectTokens)));
  const int64_t step = p.T * row_stride;
  const int side = p.E < 256 ? 256 / p.E : 1;               // tokens side by side
  float* score = smem + warp * 2 * p.E;
  if (J == 1 || tokens <= (J >= 16 ? 2 : 1) * side) {       // J == 1: eight tokens always fit
    const int k0 = p.E < 256 ? static_cast<int>(threadIdx.x) / p.E : 0;
    if (k0 < side) {
#pragma unroll 1
      for (int e = threadIdx.x - k0 * p.E; e < p.E; e += 256) {
#pragma unroll 1
        for (int k = k0; k < tokens; k += side) {
          const float* src = partials + (t0 + k) * row_stride + e;
          float v = 0.f;
#pragma unroll 1
          for (int s0 = 0; s0 < nsplit; s0 += 8, src += 8 * step) {
            float x[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) x[s] = s0 + s < nsplit ? src[s * step] : 0.f;
#pragma unroll
            for (int s = 0; s < 8; ++s) v += x[s];           // past the last split: + 0, which changes nothing
          }
          smem[k * 2 * p.E + e] = p.scoring == 1 ? v : sigmoid_score(v);
        }
      }
    }
    __syncthreads();
    if (warp >= tokens) return;
  } else {
    if (warp >= tokens) return;
    constexpr int S = J == 32 ? 1 : 4;                      // splits in flight (32 experts a lane, 4096 tokens: 70 us, 97 with two)
    const float* src = partials + (t0 + warp) * row_stride + lane;
    float v[J];
#pragma unroll
    for (int j = 0; j < J; ++j) v[j] = 0.f;
#pragma unroll 1
    for (int s0 = 0; s0 < nsplit; s0 += S, src += S * step) {
      float x[S][J];
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < J; ++j) x[s][j] = s0 + s < nsplit && lane + 32 * j < p.E ? src[s * step + 32 * j] : 0.f;
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < J; ++j) v[j] += x[s][j];
    }
#pragma unroll
    for (int j = 0; j < J; ++j) if (lane + 32 * j < p.E) score[lane + 32 * j] = p.scoring == 1 ? v[j] : sigmoid_score(v[j]);
    __syncwarp();
  }
  if (p.scoring == 1) { softmax_scores(score, p.E); __syncwarp(); }
  select_token<J>(p, t0 + warp, score, score + p.E);
}

constexpr size_t kTiledSmem = sizeof(float) * (kTM * kLd + kMaxE * kLd + kTM * kMaxE + 8 * kMaxE);

template <typename T>
static int launch_router(const T* x, const RouterParams& p, cudaStream_t st) {
  if (p.E <= 32) {
    const unsigned grid = static_cast<unsigned>((p.T + 7) / 8);
    router_small_kernel<T><<<grid, 256, 0, st>>>(x, p);
  } else {
    // more than 48 KB of dynamic shared memory needs the opt-in (per device, cheap)
    cudaFuncSetAttribute(router_tiled_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(kTiledSmem));
    const unsigned grid = static_cast<unsigned>((p.T + kTM - 1) / kTM);
    router_tiled_kernel<T><<<grid, 256, kTiledSmem, st>>>(x, p);
  }
  return check_launch("router_topk");
}

}  // namespace b200moe

using namespace b200moe;

extern "C" int b200moe_router_topk(const void* x, int x_dtype, const float* w, const float* bias,
                                   int64_t T, int64_t H, int E, int top_k, int n_group,
                                   int topk_group, int scoring, int norm_topk_prob,
                                   float routed_scaling_factor, int64_t* topk_idx,
                                   float* topk_weight, void* stream) {
  B200MOE_REQUIRE(x && w && topk_idx && topk_weight, B200MOE_BAD_ARG, "router_topk: null pointer");
  B200MOE_REQUIRE(T >= 0 && H > 0 && H % 8 == 0, B200MOE_BAD_SHAPE, "router_topk: H=%lld must be a positive multiple of 8", (long long)H);
  B200MOE_REQUIRE(E >= 1 && E <= kMaxE, B200MOE_BAD_SHAPE, "router_topk: E=%d not in [1,%d]", E, kMaxE);
  B200MOE_REQUIRE(top_k >= 1 && top_k <= kMaxTopK && top_k <= E, B200MOE_BAD_SHAPE, "router_topk: top_k=%d", top_k);
  B200MOE_REQUIRE(n_group >= 1 && n_group <= 32 && E % n_group == 0, B200MOE_BAD_SHAPE,
                  "router_topk: n_group=%d must divide E=%d and be <= 32", n_group, E);
  B200MOE_REQUIRE(topk_group >= 1 && topk_group <= n_group, B200MOE_BAD_SHAPE, "router_topk: topk_group=%d", topk_group);
  B200MOE_REQUIRE(n_group == 1 || E / n_group >= 2, B200MOE_BAD_SHAPE,
                  "router_topk: groups of %d expert(s) cannot supply a top-2 sum", E / n_group);
  B200MOE_REQUIRE(scoring == 0 || scoring == 1, B200MOE_BAD_ARG,
                  "router_topk: insupportable scoring function for MoE gating: %d", scoring);
  B200MOE_REQUIRE(aligned(x, 16) && aligned(w, 16), B200MOE_BAD_ALIGN, "router_topk: x and w must be 16-byte aligned");
  if (T == 0) return B200MOE_OK;
  RouterParams p{w, bias, T, H, E, top_k, n_group, topk_group, scoring, norm_topk_prob,
                 routed_scaling_factor, topk_idx, topk_weight};
  cudaStream_t st = as_stream(stream);
  switch (x_dtype) {
    case B200MOE_F32: return launch_router(static_cast<const float*>(x), p, st);
    case B200MOE_F16: return launch_router(static_cast<const __half*>(x), p, st);
    case B200MOE_BF16: return launch_router(static_cast<const __nv_bfloat16*>(x), p, st);
    default: return fail(B200MOE_BAD_DTYPE, "router_topk: x dtype %d", x_dtype);
  }
}

extern "C" int b200moe_router_select(const float* partials, int nsplit, int64_t partials_row_stride,
                                     const float* bias, int64_t T, int E,
                                     int top_k, int n_group, int topk_group, int scoring,
                                     int norm_topk_prob, float routed_scaling_factor, int64_t* topk_idx,
                                     float* topk_weight, void* stream) {
  B200MOE_REQUIRE(partials && topk_idx && topk_weight, B200MOE_BAD_ARG, "router_select: null pointer");
  B200MOE_REQUIRE(nsplit >= 1 && T >= 0 && E >= 1 && E <= 1024 && partials_row_stride >= E, B200MOE_BAD_SHAPE,
                  "router_select: nsplit=%d E=%d row stride %lld", nsplit, E, (long long)partials_row_stride);
  B200MOE_REQUIRE(top_k >= 1 && top_k <= kMaxTopK && top_k <= E, B200MOE_BAD_SHAPE, "router_select: top_k=%d", top_k);
  B200MOE_REQUIRE(n_group >= 1 && n_group <= 32 && E % n_group == 0 && topk_group >= 1 && topk_group <= n_group &&
                  (n_group == 1 || E / n_group >= 2), B200MOE_BAD_SHAPE, "router_select: n_group=%d topk_group=%d", n_group, topk_group);
  B200MOE_REQUIRE(scoring == 0 || scoring == 1, B200MOE_BAD_ARG,
                  "router_select: insupportable scoring function for MoE gating: %d", scoring);
  if (T == 0) return B200MOE_OK;
  RouterParams p{nullptr, bias, T, 0, E, top_k, n_group, topk_group, scoring, norm_topk_prob,
                 routed_scaling_factor, topk_idx, topk_weight};
  const unsigned grid = static_cast<unsigned>((T + 7) / 8);
  const size_t smem = sizeof(float) * kSelectTokens * 2 * E;
  if (E > 512)
    if (int rc = set_dynamic_smem(reinterpret_cast<const void*>(router_select_kernel<32>), sizeof(float) * kSelectTokens * 2 * 1024)) return rc;
  const auto kernel = E <= 32 ? router_select_kernel<1> : E <= 256 ? router_select_kernel<8>
                    : E <= 512 ? router_select_kernel<16> : router_select_kernel<32>;
  return launch_dependent("router_select", kernel, dim3(grid), 256, smem, as_stream(stream), partials, nsplit, partials_row_stride, p);
}
