// Grouped fp8 blockwise GEMM for few rows per group (decode), semantics of gemm_fp8.cu.
//
// What bounds it: the weights, one byte each, streamed once from HBM.  The 128-token tiles of gemm_fp8.cu spend
// 900-1100 SM cycles of tensor-core and promotion time on every 32 KB K block whatever the row count, more than the
// 740 cycles that a K block takes at the chip's copy rate.  Here the weights are the M = 128 rows of the MMA and the
// tokens its N = 16..64 columns, so that work shrinks with the rows: a promotion thread owns one output channel of each
// of the tile's two 128-channel halves and one accumulator per token.  Measured on 32 experts of a DeepSeek-V3 layer, 8 rows
// each (gate/up N 4096 K 7168, 940 MB of weights, then down N 7168 K 2048, 470 MB): 223 + 121 us with 128-token tiles,
// 176 + 107 us here, launch included; 153 + 85 us under the profiler = 6.1 and 5.5 TB/s.  A whole layer of 77 tokens
// (10.2 GB of weights and scales) takes 1.60 to 1.64 ms, 0.95 to 0.98 of the chip's copy rate.
//
// One persistent CTA per SM, 256 threads:
//   warp 0     TMA producer: two 128-channel x 128 B weight boxes and one token box (16/32/64 rows) per K block, 5 slots
//   warp 1     owns TMEM (4 stages x 2 halves x 64 f32 columns), issues 2 x 4 tcgen05.mma.kind::f8f6f4 (M128, N = tokens)
//   warp 3     the K block's scales a_s[token] * b_s[half], one slot per TMEM stage, fetched four K blocks ahead
//   warps 4-7  promotion (acc += dot * scale, one FMA per value as in gemm_fp8.cu: same bits) and the tile epilogue
//
// Tiles are dealt round robin, the chunks of one group and channel tile next to each other.
//
// Every wait is a bounded mbarrier wait; on expiry the kernel drains its copies, frees TMEM, writes
// B200MOE_DEVICE_TIMEOUT to the status word and returns.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "epilogue.cuh"
#include "gemm_rows.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"
#include "w4_common.cuh"

namespace b200moe {
namespace rows {

constexpr int kStages = 5, kAccStages = 4;
constexpr uint32_t kWBytes = 2 * 128 * 128;        // two halves of 128 channels x 128 B
constexpr uint32_t kTBytes = kRowsChunk * 128;     // 64 token rows x 128 B
constexpr uint32_t kSlot = kWBytes + kTBytes;
constexpr int kThreads = 256, kPromoWarp0 = 4, kPromoWarps = 4;
static_assert(int64_t(kMaxRowsPerGroup) * w4::kMaxGroups / kRowsChunk + w4::kMaxGroups < 65536, "chunk prefixes fit 16 bits");

struct Tail {
  uint64_t full[kStages], empty[kStages];
  uint64_t x_full[kAccStages];
  uint64_t tmem_full[kAccStages], tmem_empty[kAccStages];
  uint64_t promo_bar;                                        // meeting point of the promotion warps (bounded, unlike bar.sync)
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) float tscale[kAccStages][2][kRowsChunk];       // a_s[token] * b_s of each half
  alignas(16) float stage[16][256];                          // epilogue: [token][channel]
  int32_t seg[w4::kMaxGroups + 1];
  uint16_t pref[w4::kMaxGroups + 1];                         // exclusive prefix of token chunks per group
};
constexpr size_t kSmem = 1024 + size_t(kStages) * kSlot + sizeof(Tail);
static_assert(kSmem <= 232448, "shared memory of one CTA");

struct Params {
  const float* a_s; int64_t a_s_stride;
  const float* b_s;               // [W, N/128, K/128]
  void* c; int64_t c_stride;      // bytes
  float* c_s; int64_t c_s_stride; // floats
  const int64_t* seg; const int64_t* widx;
  int64_t M_total;
  int N, K, num_groups, c_dtype, fused, act;
  int32_t* status;
};

struct Tile { int m0, rows, tn, expert, ct; };

__device__ __forceinline__ Tile decode(const Tail* sh, const Params& p, int t, int num_ct) {
  // chunks of one group and channel tile are neighbours: they run at the same time and share the weights in L2
  int lo = 0, hi = p.num_groups;                       // last g with pref[g] * num_ct <= t
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (sh->pref[mid] * num_ct <= t) lo = mid; else hi = mid;
  }
  const int chunks = sh->pref[lo + 1] - sh->pref[lo];
  const int rem = t - sh->pref[lo] * num_ct;
  Tile tl;
  tl.ct = rem / chunks;
  tl.m0 = sh->seg[lo] + (rem - tl.ct * chunks) * kRowsChunk;
  tl.rows = min(kRowsChunk, sh->seg[lo + 1] - tl.m0);
  tl.tn = (tl.rows + 15) & ~15;
  tl.expert = p.widx ? static_cast<int>(p.widx[lo]) : lo;
  return tl;
}

__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag));
}

// Rows [m0, m0 + 16) of the tile from the stage to memory; a warp owns whole rows.  Not inlined: inside the K loop's
// function its registers and instructions slowed every tile down.
__device__ __noinline__ void emit(const Tail* sh, const Params& p, const Tile tl, int n0, int n1, int m0) {
  const int q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  for (int m = m0 + q; m < min(tl.rows, m0 + 16); m += kPromoWarps) {
    const float4 v0 = *reinterpret_cast<const float4*>(&sh->stage[m - m0][lane * 4]);
    const float4 v1 = *reinterpret_cast<const float4*>(&sh->stage[m - m0][128 + lane * 4]);
    uint8_t* row = static_cast<uint8_t*>(p.c) + static_cast<int64_t>(tl.m0 + m) * p.c_stride;
    if (!p.fused) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float4 v = half ? v1 : v0;
        const int n = (half ? n1 : n0) + lane * 4;
        if (n >= p.N) continue;
        if (p.c_dtype == B200MOE_F32) *reinterpret_cast<float4*>(row + n * 4) = v;
        else if (p.c_dtype == B200MOE_BF16) {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
          *reinterpret_cast<uint2*>(row + n * 2) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
          const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
          *reinterpret_cast<uint2*>(row + n * 2) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        }
      }
    } else {
      // act(gate) * up with the roundings of the unfused chain, then the 1x128 e4m3 quantizer, as in gemm_fp8.cu
      const float g[4] = {v0.x, v0.y, v0.z, v0.w}, u[4] = {v1.x, v1.y, v1.z, v1.w};
      float h[4], amax = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        h[i] = bf16r(bf16r(gate_act(bf16r(g[i]), p.act)) * bf16r(u[i]));
        amax = fmaxf(amax, fabsf(h[i]));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      const float scale = __fdiv_rn(amax, 448.f), inv = __frcp_rn(scale);
      float y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { const float r = h[i] * inv; y[i] = fmaf(fmaf(-r, scale, h[i]), inv, r); }
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(y[0], y[1]), __NV_SATFINITE, __NV_E4M3);
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(y[2], y[3]), __NV_SATFINITE, __NV_E4M3);
      *reinterpret_cast<uint32_t*>(row + tl.ct * 128 + lane * 4) = lo | (hi << 16);
      if (lane == 0) p.c_s[static_cast<int64_t>(tl.m0 + m) * p.c_s_stride + tl.ct] = scale;
    }
  }
}

template <int N, typename F>
__device__ __forceinline__ void for_blocks(F&& f) {
  f(std::integral_constant<int, 0>{});
  if constexpr (N > 1) f(std::integral_constant<int, 1>{});
  if constexpr (N > 2) f(std::integral_constant<int, 2>{});
  if constexpr (N > 3) f(std::integral_constant<int, 3>{});
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_fp8_rows_kernel(const __grid_constant__ w4::RowMaps tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Tail* sh = reinterpret_cast<Tail*>(smem + size_t(kStages) * kSlot);
  volatile int* abort_flag = &sh->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KB = p.K / 128, NB = p.N / 128;
  const int num_ct = p.fused ? NB / 2 : (p.N + 255) / 256;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { ptx::mbar_init(&sh->full[s], 1); ptx::mbar_init(&sh->empty[s], 1); }
    for (int s = 0; s < kAccStages; ++s) {
      ptx::mbar_init(&sh->x_full[s], 1); ptx::mbar_init(&sh->tmem_full[s], 1); ptx::mbar_init(&sh->tmem_empty[s], kPromoWarps);
    }
    ptx::mbar_init(&sh->promo_bar, kPromoWarps);
    sh->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
#pragma unroll
    for (int i = 0; i < 3; ++i) ptx::prefetch_tensormap(&tmap_a.m[i]);
    ptx::prefetch_tensormap(&tmap_b);
  }
  if (warp == 1) {
    ptx::tmem_alloc<1>(&sh->tmem_base, w4::kTmemCols);
    ptx::tmem_relinquish<1>();
  }
  // the setup above overlaps the tail of the kernel before; from here on its results are read
  wait_for_predecessors();
  for (int g = threadIdx.x; g <= p.num_groups; g += kThreads)
    sh->seg[g] = p.seg ? static_cast<int32_t>(p.seg[g]) : (g == 0 ? 0 : static_cast<int32_t>(p.M_total));
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  if (warp == 2) {
    int run = 0;
    for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
      const int g = g0 + lane;
      int v = 0;
      if (g < p.num_groups) { const int m = sh->seg[g + 1] - sh->seg[g]; v = m > 0 ? (m + kRowsChunk - 1) / kRowsChunk : 0; }
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
      if (g < p.num_groups) sh->pref[g] = static_cast<uint16_t>(run + incl - v);
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) sh->pref[p.num_groups] = static_cast<uint16_t>(run);
  }
  __syncthreads();
  const uint32_t tmem_base = sh->tmem_base;
  const int total = sh->pref[p.num_groups] * num_ct, first = static_cast<int>(blockIdx.x), step = static_cast<int>(gridDim.x);
  // first output channel of the tile's two halves (within the expert's N channels)
  auto half_ch = [&](const Tile& tl, int& n0, int& n1) {
    n0 = p.fused ? tl.ct * 128 : tl.ct * 256;
    n1 = p.fused ? p.N / 2 + tl.ct * 128 : n0 + 128;
  };

  if (warp == 0 && ptx::elect_one()) {
    // ---- weights and token rows ------------------------------------------------------------------------------------
    int stage = 0; uint32_t phase = 0;
    w4::Armed armed;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = decode(sh, p, t, num_ct);
      const int sel = tl.tn <= 16 ? 0 : (tl.tn <= 32 ? 1 : 2);
      int n0, n1;
      half_ch(tl, n0, n1);
      const bool second = n1 < p.N;
      const uint32_t bytes = (second ? kWBytes : kWBytes / 2) + (16u << sel) * 128u;
      const int row0 = tl.expert * p.N + n0, row1 = tl.expert * p.N + n1;
      for (int kb = 0; kb < KB; ++kb) {
        if (!ptx::mbar_wait(&sh->empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
        uint8_t* sw = smem + size_t(stage) * kSlot;
        ptx::mbar_arrive_expect_tx(&sh->full[stage], bytes);
        armed.arm(stage, phase);
        ptx::tma_load_2d(sw, &tmap_b, &sh->full[stage], kb * 128, row0);
        if (second) ptx::tma_load_2d(sw + kWBytes / 2, &tmap_b, &sh->full[stage], kb * 128, row1);
        ptx::tma_load_2d(sw + kWBytes, &tmap_a.m[sel], &sh->full[stage], kb * 128, tl.m0);
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
    if (!ok) armed.drain(sh->full, kStages);
  } else if (warp == 1 && ptx::elect_one()) {
    // ---- MMA issuer: channels are the M = 128 rows, tokens the N columns -------------------------------------------
    int st = 0, as = 0;
    uint32_t ph = 0, pacc = 0;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = decode(sh, p, t, num_ct);
      const uint32_t idesc = ptx::umma_idesc(1, 0, 0, 128, static_cast<uint32_t>(tl.tn));
      for (int kb = 0; kb < KB; ++kb) {
        // x_full: the scales of this K block are in place, so that the promotion warps wait for tmem_full alone
        if (!ptx::mbar_wait(&sh->tmem_empty[as], pacc ^ 1u, abort_flag) || !ptx::mbar_wait(&sh->x_full[as], pacc, abort_flag) ||
            !ptx::mbar_wait(&sh->full[st], ph, abort_flag)) { ok = false; break; }
        ptx::tc_fence_after_sync();
        const uint32_t d = tmem_base + static_cast<uint32_t>(as) * 128u;
        const uint32_t sw = ptx::smem_u32(smem + size_t(st) * kSlot);
        const uint64_t wdesc = ptx::umma_desc_sw128(sw), tdesc = ptx::umma_desc_sw128(sw + kWBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k) {      // halves alternate: an instruction does not wait for the one that feeds its accumulator
          ptx::umma_f8f6f4<1>(d, wdesc + 2 * k, tdesc + 2 * k, idesc, k > 0 ? 1u : 0u);
          ptx::umma_f8f6f4<1>(d + 64u, wdesc + (kWBytes / 2 >> 4) + 2 * k, tdesc + 2 * k, idesc, k > 0 ? 1u : 0u);
        }
        ptx::umma_commit(&sh->empty[st]);
        ptx::umma_commit(&sh->tmem_full[as]);
        if (++st == kStages) { st = 0; ph ^= 1u; }
        if (++as == kAccStages) { as = 0; pacc ^= 1u; }
      }
    }
  } else if (warp == 3) {
    // ---- scales ----------------------------------------------------------------------------------------------------
    int as = 0;
    uint32_t pacc = 0;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = decode(sh, p, t, num_ct);
      const bool two = tl.tn > 32;
      const int64_t last = p.M_total - 1;
      int n0, n1;
      half_ch(tl, n0, n1);
      if (n1 >= p.N) n1 = n0;
      const float* src[4] = {p.a_s + min(static_cast<int64_t>(tl.m0 + lane), last) * p.a_s_stride,
                             p.a_s + min(static_cast<int64_t>(tl.m0 + lane + 32), last) * p.a_s_stride,
                             p.b_s + (static_cast<int64_t>(tl.expert) * NB + (n0 >> 7)) * KB,
                             p.b_s + (static_cast<int64_t>(tl.expert) * NB + (n1 >> 7)) * KB};
      // requested four K blocks ahead of their use: a load consumed in the same step would put an L2 or HBM round trip
      // into every K block
      float nxt[4][4];
      auto fetch = [&](int kb0) {
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
          for (int u = 0; u < 4; ++u) nxt[v][u] = (kb0 + u < KB && (v != 1 || two)) ? __ldg(src[v] + kb0 + u) : 0.f;
      };
      fetch(0);
      for (int kb0 = 0; ok && kb0 < KB; kb0 += 4) {
        float cur[4][4];
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
          for (int u = 0; u < 4; ++u) cur[v][u] = nxt[v][u];
        fetch(kb0 + 4);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (kb0 + u >= KB) break;
          if (!warp_wait(&sh->tmem_empty[as], pacc ^ 1u, abort_flag)) { ok = false; break; }
          sh->tscale[as][0][lane] = cur[0][u] * cur[2][u];
          sh->tscale[as][1][lane] = cur[0][u] * cur[3][u];
          if (two) {
            sh->tscale[as][0][lane + 32] = cur[1][u] * cur[2][u];
            sh->tscale[as][1][lane + 32] = cur[1][u] * cur[3][u];
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&sh->x_full[as]);
          if (++as == kAccStages) { as = 0; pacc ^= 1u; }
        }
      }
    }
  } else if (warp >= kPromoWarp0) {
    // ---- promotion and epilogue: thread = output channel (one of each half), registers = tokens ----------------------
    const int q = warp & 3, c = q * 32 + lane;            // TMEM lane = channel within the half
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    int as = 0;
    uint32_t pacc = 0, meet = 0;
    bool ok = true;
    auto promo_sync = [&]() {
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh->promo_bar);
      ok = warp_wait(&sh->promo_bar, meet, abort_flag);
      meet ^= 1u;
      return ok;
    };
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = decode(sh, p, t, num_ct);
      int n0, n1;
      half_ch(tl, n0, n1);
      // the K loop exists once per number of 16-token blocks: short straight code
      auto tile_body = [&](auto nblocks) {
        constexpr int kBlocks = decltype(nblocks)::value;
        float acc0[kBlocks * 16], acc1[kBlocks * 16];
#pragma unroll
        for (int m = 0; m < kBlocks * 16; ++m) { acc0[m] = 0.f; acc1[m] = 0.f; }
        for (int kb = 0; kb < KB; ++kb) {
          if (!warp_wait(&sh->tmem_full[as], pacc, abort_flag)) { ok = false; return; }
          ptx::tc_fence_after_sync();
          const uint32_t tcol = tmem_base + lane_base + static_cast<uint32_t>(as) * 128u;
          uint32_t d0[16], d1[16];
          ptx::tmem_ld16(tcol, d0);
          ptx::tmem_ld16(tcol + 64, d1);
          const ulonglong2* s0p = reinterpret_cast<const ulonglong2*>(sh->tscale[as][0]);
          const ulonglong2* s1p = reinterpret_cast<const ulonglong2*>(sh->tscale[as][1]);
#pragma unroll
          for (int mb = 0; mb < kBlocks; ++mb) {
            ulonglong2 s0[4], s1[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { s0[j] = s0p[mb * 4 + j]; s1[j] = s1p[mb * 4 + j]; }
            ptx::tmem_ld_wait16(d0, d1);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              ptx::ffma2(acc0[mb * 16 + j * 4], acc0[mb * 16 + j * 4 + 1], d0[j * 4], d0[j * 4 + 1], s0[j].x);
              ptx::ffma2(acc0[mb * 16 + j * 4 + 2], acc0[mb * 16 + j * 4 + 3], d0[j * 4 + 2], d0[j * 4 + 3], s0[j].y);
            }
            if (mb + 1 < kBlocks) ptx::tmem_ld16(tcol + (mb + 1) * 16, d0);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              ptx::ffma2(acc1[mb * 16 + j * 4], acc1[mb * 16 + j * 4 + 1], d1[j * 4], d1[j * 4 + 1], s1[j].x);
              ptx::ffma2(acc1[mb * 16 + j * 4 + 2], acc1[mb * 16 + j * 4 + 3], d1[j * 4 + 2], d1[j * 4 + 3], s1[j].y);
            }
            if (mb + 1 < kBlocks) ptx::tmem_ld16(tcol + 64 + (mb + 1) * 16, d1);
          }
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&sh->tmem_empty[as]);
          if (++as == kAccStages) { as = 0; pacc ^= 1u; }
        }

        // The epilogue goes through a [16 tokens][256 channels] f32 stage in shared memory, so that only the copy into the
        // stage is unrolled over the accumulators: the rest is short loops in which a warp owns whole tokens.  (Unrolled
        // over up to 128 registers the epilogue was several thousand instructions that each CTA of a small problem
        // fetches once: 5 us.)
        auto dump = [&](auto block) {
          constexpr int m0 = decltype(block)::value * 16;
#pragma unroll
          for (int m = 0; m < 16; ++m) { sh->stage[m][c] = acc0[m0 + m]; sh->stage[m][128 + c] = acc1[m0 + m]; }
        };
        for_blocks<kBlocks>([&](auto block) {
          if (!ok) return;
          dump(block);
          if (!promo_sync()) return;
          emit(sh, p, tl, n0, n1, decltype(block)::value * 16);
          promo_sync();                                   // the stage may be overwritten
        });
      };
      switch (tl.tn >> 4) {
        case 1: tile_body(std::integral_constant<int, 1>{}); break;
        case 2: tile_body(std::integral_constant<int, 2>{}); break;
        case 3: tile_body(std::integral_constant<int, 3>{}); break;
        default: tile_body(std::integral_constant<int, 4>{}); break;
      }
    }
  }

  // ---- teardown ------------------------------------------------------------------------------------------------
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc<1>(tmem_base, w4::kTmemCols);
  if (threadIdx.x == 0 && sh->abort_flag && p.status) *p.status = B200MOE_DEVICE_TIMEOUT;
}

int launch_fp8(const void* a, int64_t a_stride, const float* a_s, int64_t a_s_stride, const void* b, const float* b_s, void* c,
               int c_dtype, int64_t c_stride, float* c_s, int64_t c_s_stride, int64_t M_total, int64_t N, int64_t K, int num_groups,
               int num_weights, const int64_t* seg, const int64_t* widx, int fused, int act, int32_t* status, cudaStream_t st) {
  int sms = 0;
  if (int rc = require_sm100(&sms)) return rc;
  w4::RowMaps ma;
  CUtensorMap mb;
  for (int i = 0; i < 3; ++i)
    if (int rc = cached_tensor_map_u8(&ma.m[i], a, static_cast<uint64_t>(M_total), static_cast<uint64_t>(K),
                                      static_cast<uint64_t>(a_stride), 16u << i)) return rc;
  ma.m[3] = ma.m[2];
  if (int rc = cached_tensor_map_u8(&mb, b, static_cast<uint64_t>(num_weights) * N, static_cast<uint64_t>(K),
                                    static_cast<uint64_t>(K), 128)) return rc;
  Params p{a_s, a_s_stride, b_s, c, c_stride, c_s, c_s_stride, seg, widx, M_total, static_cast<int>(N), static_cast<int>(K),
           num_groups, c_dtype, fused, act, status};
  if (int rc = set_dynamic_smem(reinterpret_cast<const void*>(gemm_fp8_rows_kernel), kSmem)) return rc;
  return launch_dependent("gemm_fp8_rows_kernel", gemm_fp8_rows_kernel, dim3(static_cast<unsigned>(sms)), kThreads, kSmem, st, ma, mb, p);
}

}  // namespace rows
}  // namespace b200moe
