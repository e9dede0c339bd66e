// Grouped w4a8 GEMM for few rows per expert (decode, small prefill batches), with the int4 weights unpacked inside the kernel
// and the weights, not the tokens, on the 128-row side of the tensor-core tile.
//
//   reference: w4a8_gemm_kernel (quantization/w4a8_kernel.py:317-404) unpacks the nibbles, applies
//   (q - z4) * s4 and feeds the int8 dot product inside its K loop (:362-380); per K block
//   acc += float(dot in s32) * a_s[m,kb] * b_s[n/128,kb].  The grouped form follows grouped_gemm_triton
//   (moe/group_gemm_kernel.py:291-513).
//
// Three moves keep the per-weight work of the CUDA cores small in the decode regime:
//   * The dot product of a token row a with w8 = (q - z) * s over one 128-wide K block (one (s, z) per output channel
//     and K block) is  s * (a . q  -  z * sum_k a_k).  So the tensor core multiplies the int8 tokens with the RAW
//     nibbles q (0..15 as int8) and the promotion restores the exact integer with exact f32 arithmetic.
//     This equals the reference's int8 product whenever (q - z) * s fits int8 for every nibble q the weight holds,
//     which its quantizer guarantees (quantization/w4a8_kernel.py:228-262); the Python layer checks it once per
//     weight (smallest and largest nibble of every scale group) and otherwise expands the weight to int8.
//   * Output channels are the M = 128 rows of the MMA and the tokens its N = 16..64 columns: a thread of the promotion
//     warps owns one channel, keeps that channel's (s, z) in registers and touches only as many accumulators as there
//     are tokens, so the per-K-block work of the CUDA cores shrinks with the batch instead of staying at 128 x 256.
//   * The weight operand lives in tensor memory.  A packed word holds 8 channels at one k, the operand wants four k of one
//     channel per 32-bit column: the converters transpose bytes in registers and store with the one tcgen05.st shape whose
//     register layout fits, 0.7 instructions per weight and no shared-memory write or MMA read of the operand.
//
// What bounds it: issue slots (62 % at 16 rows per expert), first of the conversion, from about 32 rows on of the promotion.
// 64 experts, gate/up N 4096 K 7168 then down N 7168 K 2048, us (operand in shared memory,
// roles entered by lane == 0, four promotion warps with integer multiply-adds -> here): 1 row per expert 338 + 186 -> 218 +
// 129, 16 rows 358 + 189 -> 221 + 131 (4.4 TB/s of packed weights), 48 rows 566 + 291 -> 355 + 210, 64 rows 690 + 377 ->
// 416 + 244, 94 rows 1100 + 606 -> 706 + 384, 256 rows 2845 + 1491 -> 1643 + 897.
//
// One persistent CTA per SM, 640 threads (the roles that are one thread are entered through elect.sync: under `lane == 0`
// each tcgen05 instruction took about 90 cycles to issue):
//   warp 0       TMA producer of the packed weights: per K block two boxes of 16 packed rows x 128 k (int32 words, 8 output
//                channels per word, quantization/bitpack.py:9-36; 128-byte swizzle so that the converters read without
//                bank conflicts), 16 KB per K block, 6-slot ring
//   warp 2       TMA producer of the int8 token rows (box of 16/32/64 rows x 128 B) and of the tile's 2 x 128 (s4, z4)
//                pairs (two 256-byte bulk copies), 7-slot ring
//   warp 3       per K block and token: sum of the 128 int8 values (dp4a) and the token's scale times the two
//                block scales, written beside the token stage
//   warps 12-19  converters: packed words -> int8 nibbles in the tensor-memory operand (2 stages of 64 columns)
//   warp 1       owns TMEM (2 operand stages, 3 stages of 128 s32 accumulator columns); per K block 2 x 4
//                tcgen05.mma.kind::i8 (M128, N = tokens, K32)
//   warps 4-11   promotion (one channel per thread) and the tile epilogue
//
// Every wait is a bounded mbarrier wait; on expiry the kernel drains its copies, frees TMEM, writes
// B200MOE_DEVICE_TIMEOUT to the status word and returns.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "epilogue.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"
#include "w4_common.cuh"

namespace b200moe {
namespace w4 {

constexpr int kChunk = 64;                       // tokens per tile at most
constexpr int kPStages = 6, kOpStages = 2, kTStages = 7, kAccStages = 3;
constexpr uint32_t kPBytes = 32 * 128 * 4;       // 32 packed rows x 128 words
constexpr uint32_t kTBytes = kChunk * 128;       // 64 token rows x 128 B
constexpr uint32_t kOpCols = 64;                 // tensor-memory columns of one weight operand: 2 halves x 128 k
constexpr uint32_t kAccCol = kOpStages * kOpCols;
static_assert(kAccCol + kAccStages * 2 * kChunk <= kTmemCols, "tensor memory");
constexpr int kThreads8 = 640;
constexpr int kPromoWarp0 = 4, kPromoWarps = 8, kConvWarp0 = 12, kConvWarps8 = 8;
// Register hand-over: the kernel starts with 96 registers per thread; the promotion warps may only grow by what the
// converters of the same CTA have released (an increase beyond that would wait forever).
constexpr int kRegsLaunch = 96, kRegsConv = 56, kRegsPromo = 136;
static_assert(kThreads8 * kRegsLaunch <= 65536 &&
              (kRegsLaunch - kRegsConv) * kConvWarps8 >= (kRegsPromo - kRegsLaunch) * kPromoWarps, "setmaxnreg budget");

struct Tail8 {
  uint64_t p_full[kPStages], p_empty[kPStages];
  uint64_t op_full[kOpStages], op_empty[kOpStages];
  uint64_t t_full[kTStages], t_empty[kTStages];
  uint64_t x_full[kTStages];                     // the token stage's sums and scales have been written
  uint64_t tmem_full[kAccStages], tmem_empty[kAccStages];
  uint64_t stage_full, stage_free;               // fused epilogue: the bf16 stage has been written / read
  uint32_t tmem_base;
  int abort_flag;
  // travelling with a token stage (one K block):
  alignas(16) float rsum[kTStages][kChunk];      // sum of the token's 128 int8 values
  alignas(16) float tscale[kTStages][2][kChunk]; // the token's scale times the scale of each 128-channel block
  alignas(16) uint16_t sz[kTStages][256];        // (s4, z4) of the tile's 2 x 128 channels (bulk copies)
  alignas(16) __nv_bfloat16 stage[kChunk][256];  // fused epilogue: gate and up of one tile, [token][channel]
  int32_t seg[kMaxGroups + 1];
  int32_t pref[kMaxGroups + 1];                  // exclusive prefix of token chunks per group
};
constexpr size_t kRing8 = size_t(kTStages) * kTBytes + size_t(kPStages) * kPBytes;
constexpr size_t kSmem8 = 1024 + kRing8 + sizeof(Tail8);
static_assert(kSmem8 <= 232448, "shared memory of one CTA");

struct Params8 {
  const float* a_s; int64_t a_s_stride;
  const float* b_s;               // [W, N/128, K/128]
  const uint16_t* sz_t;           // [W, K/128, N]: (s4, z4) int8 pairs, s4 in the low byte
  void* c; int64_t c_stride;      // bytes
  float* c_s; int64_t c_s_stride; // floats
  const int64_t* seg; const int64_t* widx;
  int64_t M_total;
  int N, K, num_groups, c_dtype, fused, act;
  int32_t* status;
};

struct Tile8 { int m0, rows, tn, expert, ct; };

__device__ __forceinline__ Tile8 decode_tile8(const Tail8* sh, const Params8& p, int t, int num_ct) {
  const int mc = t / num_ct;
  int lo = 0, hi = p.num_groups;           // last g with pref[g] <= mc
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (sh->pref[mid] <= mc) lo = mid; else hi = mid;
  }
  Tile8 tl;
  tl.m0 = sh->seg[lo] + (mc - sh->pref[lo]) * kChunk;
  tl.rows = min(kChunk, sh->seg[lo + 1] - tl.m0);
  tl.tn = (tl.rows + 15) & ~15;
  tl.expert = p.widx ? static_cast<int>(p.widx[lo]) : lo;
  tl.ct = t - mc * num_ct;
  return tl;
}

// Packed row (of a lane quarter's eight) that the threads u = lane / 4 of a converter warp read: neighbours u are rows 4
// apart, whose 16-byte chunks the swizzle puts into different halves of the banks.
__device__ __forceinline__ int packed_row(int u) { return (u >> 1) | ((u & 1) << 2); }

// A whole warp waits for a barrier phase (every lane queries it: measured faster than one lane and a shuffle).
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag));
}

// (acc0, acc1) += (dot - z * rsum) * s * ts for two tokens.  Every step but the last is exact: dot and the sums are integers
// of at most 22 bits, so are their combinations, and the product with s is the integer dot product that the reference
// forms (rounded to f32 as an int -> float conversion would round it, if a weight leaves the int8 range).  The integer
// is made a float by adding it to the bits of 1.5 * 2^23, whose ulp is 1; nz * rsum - 1.5 * 2^23 takes that off again.
// Packed f32 instead of two integer multiply-adds and a conversion per value, which run at half and a quarter of the rate.
__device__ __forceinline__ void promote2(float& acc0, float& acc1, uint32_t d0, uint32_t d1, uint64_t rsum2, uint64_t nz2,
                                         uint64_t s2, uint64_t ts2) {
  constexpr float kMagic = 12582912.f;
  constexpr uint32_t kMagicBits = 0x4B400000u;
  const uint64_t f = ptx::pack_f32x2(__uint_as_float(d0 + kMagicBits), __uint_as_float(d1 + kMagicBits));
  const uint64_t off = ptx::fma_f32x2(nz2, rsum2, ptx::pack_f32x2(-kMagic, -kMagic));
  const uint64_t u = ptx::mul_f32x2(ptx::add_f32x2(f, off), s2);
  const uint64_t r = ptx::fma_f32x2(u, ts2, ptx::pack_f32x2(acc0, acc1));
  ptx::unpack_f32x2(r, acc0, acc1);
}

// One token of the fused epilogue: 128 gate and 128 up values of the stage -> int8 row and its scale.  128 values that are all
// NaN (a token with an infinite value) have a NaN scale, as the reference's maximum gives; act_quant gives them a scale of 0.
__device__ __forceinline__ void emit_row(const Tail8* sh, const Params8& p, const Tile8& tl, int m) {
  const int lane = threadIdx.x & 31;
  const uint2 gv = *reinterpret_cast<const uint2*>(&sh->stage[m][lane * 4]);
  const uint2 uv = *reinterpret_cast<const uint2*>(&sh->stage[m][128 + lane * 4]);
  float h[4] = {__uint_as_float(gv.x << 16), __uint_as_float(gv.x & 0xFFFF0000u),
                __uint_as_float(gv.y << 16), __uint_as_float(gv.y & 0xFFFF0000u)};
  const float up[4] = {__uint_as_float(uv.x << 16), __uint_as_float(uv.x & 0xFFFF0000u),
                       __uint_as_float(uv.y << 16), __uint_as_float(uv.y & 0xFFFF0000u)};
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = bf16r(bf16r(gate_act(h[i], p.act)) * up[i]);
  float amax = fmaxf(fmaxf(fabsf(h[0]), fabsf(h[1])), fmaxf(fabsf(h[2]), fabsf(h[3])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = __fdiv_rn(amax, 127.f);
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float rq = floorf(__fdiv_rn(h[i], scale) + 0.5f);
    packed |= (static_cast<uint32_t>(__float2int_rz(fminf(fmaxf(rq, -128.f), 127.f))) & 0xFFu) << (8 * i);
  }
  *reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(p.c) + static_cast<int64_t>(tl.m0 + m) * p.c_stride + tl.ct * 128 + lane * 4) = packed;
  if (lane == 0) p.c_s[static_cast<int64_t>(tl.m0 + m) * p.c_s_stride + tl.ct] = __half2float(__float2half_rn(scale));
}

__global__ void __launch_bounds__(kThreads8, 1)
gemm_w4a8_kernel(const __grid_constant__ RowMaps tmap_a, const __grid_constant__ CUtensorMap tmap_p, const Params8 p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_t = smem;                                          // int8 token tiles (TMA)
  uint8_t* smem_p = smem_t + size_t(kTStages) * kTBytes;           // packed words (TMA)
  Tail8* sh = reinterpret_cast<Tail8*>(smem_p + size_t(kPStages) * kPBytes);
  volatile int* abort_flag = &sh->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KB = p.K / 128, NB = p.N / 128;
  const int num_ct = p.fused ? (p.N / 2) / 128 : (p.N + 255) / 256;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPStages; ++s) { ptx::mbar_init(&sh->p_full[s], 1); ptx::mbar_init(&sh->p_empty[s], kConvWarps8); }
    for (int s = 0; s < kOpStages; ++s) { ptx::mbar_init(&sh->op_full[s], kConvWarps8); ptx::mbar_init(&sh->op_empty[s], 1); }
    for (int s = 0; s < kTStages; ++s) {
      ptx::mbar_init(&sh->t_full[s], 1); ptx::mbar_init(&sh->t_empty[s], 1 + kPromoWarps); ptx::mbar_init(&sh->x_full[s], 1);
    }
    for (int s = 0; s < kAccStages; ++s) { ptx::mbar_init(&sh->tmem_full[s], 1); ptx::mbar_init(&sh->tmem_empty[s], kPromoWarps); }
    ptx::mbar_init(&sh->stage_full, kPromoWarps); ptx::mbar_init(&sh->stage_free, kPromoWarps);
    sh->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
#pragma unroll
    for (int i = 0; i < 3; ++i) ptx::prefetch_tensormap(&tmap_a.m[i]);
    ptx::prefetch_tensormap(&tmap_p);
  }
  if (warp == 1) {
    ptx::tmem_alloc<1>(&sh->tmem_base, kTmemCols);
    ptx::tmem_relinquish<1>();
  }
  for (int g = threadIdx.x; g <= p.num_groups; g += kThreads8) sh->seg[g] = static_cast<int32_t>(p.seg[g]);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  if (warp == 3) {
    int run = 0;
    for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
      const int g = g0 + lane;
      int v = 0;
      if (g < p.num_groups) { const int m = sh->seg[g + 1] - sh->seg[g]; v = m > 0 ? (m + kChunk - 1) / kChunk : 0; }
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
      if (g < p.num_groups) sh->pref[g] = run + incl - v;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) sh->pref[p.num_groups] = run;
  }
  __syncthreads();
  const uint32_t tmem_base = sh->tmem_base;
  const int total_tiles = sh->pref[p.num_groups] * num_ct;
  const int first = static_cast<int>(blockIdx.x), step = static_cast<int>(gridDim.x);
  // first output channel of the tile's two 128-channel halves (within the expert's N channels)
  auto half_ch = [&](const Tile8& tl, int& n0, int& n1) {
    n0 = p.fused ? tl.ct * 128 : tl.ct * 256;
    n1 = p.fused ? p.N / 2 + tl.ct * 128 : n0 + 128;
  };

  if (warp < kPromoWarp0) {
    if (warp == 0 && ptx::elect_one()) {
      // ---- packed weights: per K block two boxes of 16 packed rows (128 channels) x 128 k ---------------------------
      int stage = 0; uint32_t phase = 0;
      Armed armed;
      bool ok = true;
      for (int t = first; ok && t < total_tiles; t += step) {
        const Tile8 tl = decode_tile8(sh, p, t, num_ct);
        int n0, n1;
        half_ch(tl, n0, n1);
        const int prow0 = (tl.expert * p.N + n0) >> 3, prow1 = (tl.expert * p.N + n1) >> 3;
        for (int kb = 0; kb < KB; ++kb) {
          if (!ptx::mbar_wait(&sh->p_empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
          uint8_t* sp = smem_p + size_t(stage) * kPBytes;
          ptx::mbar_arrive_expect_tx(&sh->p_full[stage], kPBytes);
          armed.arm(stage, phase);
          // boxes of 32 k x 16 packed rows x 4 k groups, 128-byte swizzle; rows past the tensor: zero fill
          ptx::tma_load_3d(sp, &tmap_p, &sh->p_full[stage], 0, prow0, kb * 4);
          ptx::tma_load_3d(sp + kPBytes / 2, &tmap_p, &sh->p_full[stage], 0, prow1, kb * 4);
          if (++stage == kPStages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) armed.drain(sh->p_full, kPStages);
    } else if (warp == 2 && ptx::elect_one()) {
      // ---- token rows and the channels' (s4, z4) pairs -------------------------------------------------------------
      int stage = 0; uint32_t phase = 0;
      Armed armed;
      bool ok = true;
      for (int t = first; ok && t < total_tiles; t += step) {
        const Tile8 tl = decode_tile8(sh, p, t, num_ct);
        const int sel = tl.tn <= 16 ? 0 : (tl.tn <= 32 ? 1 : 2);
        const uint32_t bytes = (16u << sel) * 128u + 512u;
        int n0, n1;
        half_ch(tl, n0, n1);
        if (n1 >= p.N) n1 = n0;
        const uint16_t* szp = p.sz_t + static_cast<int64_t>(tl.expert) * KB * p.N;
        for (int kb = 0; kb < KB; ++kb) {
          if (!ptx::mbar_wait(&sh->t_empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
          ptx::mbar_arrive_expect_tx(&sh->t_full[stage], bytes);
          armed.arm(stage, phase);
          ptx::tma_load_2d(smem_t + size_t(stage) * kTBytes, &tmap_a.m[sel], &sh->t_full[stage], kb * 128, tl.m0);
          ptx::bulk_load(&sh->sz[stage][0], szp + static_cast<int64_t>(kb) * p.N + n0, 256u, &sh->t_full[stage]);
          ptx::bulk_load(&sh->sz[stage][128], szp + static_cast<int64_t>(kb) * p.N + n1, 256u, &sh->t_full[stage]);
          if (++stage == kTStages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) armed.drain(sh->t_full, kTStages);
    } else if (warp == 1 && ptx::elect_one()) {
      // ---- MMA issuer: channels are the M = 128 rows, tokens the N columns ---------------------------------------
      int so = 0, st = 0, as = 0;
      uint32_t po = 0, pt = 0, pacc = 0;
      bool ok = true;
      for (int t = first; ok && t < total_tiles; t += step) {
        const Tile8 tl = decode_tile8(sh, p, t, num_ct);
        const uint32_t idesc = ptx::umma_idesc(2, 1, 1, 128, static_cast<uint32_t>(tl.tn));   // D s32, A and B signed int8
        for (int kb = 0; kb < KB; ++kb) {
          // x_full (sums written) follows t_full (tokens and pairs landed): the warp that arrives on it waited for
          // t_full.  Waiting for it here lets the promotion warps wait for tmem_full alone.
          if (!ptx::mbar_wait(&sh->x_full[st], pt, abort_flag) || !ptx::mbar_wait(&sh->tmem_empty[as], pacc ^ 1u, abort_flag) ||
              !ptx::mbar_wait(&sh->op_full[so], po, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after_sync();
          const uint32_t d = tmem_base + kAccCol + static_cast<uint32_t>(as) * (2 * kChunk);
          const uint32_t a = tmem_base + static_cast<uint32_t>(so) * kOpCols;
          const uint64_t tdesc = ptx::umma_desc_sw128(ptx::smem_u32(smem_t + size_t(st) * kTBytes));
          // 32 k are eight columns of the operand; the two halves alternate, so that an instruction does not wait for
          // the one that feeds its accumulator
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            ptx::umma_i8_ts(d, a + 8u * k, tdesc + 2 * k, idesc, k > 0 ? 1u : 0u);
            ptx::umma_i8_ts(d + kChunk, a + kOpCols / 2 + 8u * k, tdesc + 2 * k, idesc, k > 0 ? 1u : 0u);
          }
          ptx::umma_commit(&sh->op_empty[so]);
          ptx::umma_commit(&sh->t_empty[st]);
          ptx::umma_commit(&sh->tmem_full[as]);
          if (++so == kOpStages) { so = 0; po ^= 1u; }
          if (++st == kTStages) { st = 0; pt ^= 1u; }
          if (++as == kAccStages) { as = 0; pacc ^= 1u; }
        }
      }
    } else if (warp == 3) {
      // ---- per K block: each token's sum of its 128 int8 values and its scale times the two block scales, written
      //      beside the token stage for the promotion warps ----------------------------------------------------------
      int st = 0;
      uint32_t pt = 0;
      bool ok = true;
      // four K blocks of scales per 16-byte load when the rows allow it
      const bool vec = (KB & 3) == 0 && (p.a_s_stride & 3) == 0 && (reinterpret_cast<uintptr_t>(p.a_s) & 15) == 0 &&
                       (reinterpret_cast<uintptr_t>(p.b_s) & 15) == 0;
      for (int t = first; ok && t < total_tiles; t += step) {
        const Tile8 tl = decode_tile8(sh, p, t, num_ct);
        const bool two = tl.tn > 32;
        const int64_t last = p.M_total - 1;
        int n0, n1;
        half_ch(tl, n0, n1);
        if (n1 >= p.N) n1 = n0;
        const float* src[4] = {p.a_s + min(static_cast<int64_t>(tl.m0 + lane), last) * p.a_s_stride,
                               p.a_s + min(static_cast<int64_t>(tl.m0 + lane + 32), last) * p.a_s_stride,
                               p.b_s + (static_cast<int64_t>(tl.expert) * NB + (n0 >> 7)) * KB,
                               p.b_s + (static_cast<int64_t>(tl.expert) * NB + (n1 >> 7)) * KB};
        // The scales of K blocks kb + 4 .. kb + 7 are requested while kb .. kb + 3 are worked on: a load issued and
        // consumed in the same iteration would put an L2 round trip into every K block.
        float cur[4][4], nxt[4][4];
        auto fetch = [&](float (&dst)[4][4], int kb0) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (v == 1 && !two) { dst[1][0] = dst[1][1] = dst[1][2] = dst[1][3] = 0.f; continue; }
            if (vec) {
              const float4 f = __ldg(reinterpret_cast<const float4*>(src[v] + kb0));
              dst[v][0] = f.x; dst[v][1] = f.y; dst[v][2] = f.z; dst[v][3] = f.w;
            } else {
#pragma unroll
              for (int u = 0; u < 4; ++u) dst[v][u] = kb0 + u < KB ? __ldg(src[v] + kb0 + u) : 0.f;
            }
          }
        };
        fetch(nxt, 0);
        for (int kb0 = 0; ok && kb0 < KB; kb0 += 4) {
#pragma unroll
          for (int v = 0; v < 4; ++v)
#pragma unroll
            for (int u = 0; u < 4; ++u) cur[v][u] = nxt[v][u];
          if (kb0 + 4 < KB) fetch(nxt, kb0 + 4);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (kb0 + u >= KB) break;
            if (!warp_wait(&sh->t_full[st], pt, abort_flag)) { ok = false; break; }
            // A row's 16-byte chunks are permuted by the swizzle, which a sum does not see; lanes start at different
            // chunks so that the 32 rows (128 bytes apart) do not meet in the same banks.
            const uint8_t* slot = smem_t + size_t(st) * kTBytes;
            int ra[4] = {0, 0, 0, 0}, rb[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint4 v = *reinterpret_cast<const uint4*>(slot + lane * 128 + (((j + lane) & 7) << 4));
              ra[0] = __dp4a(static_cast<int>(v.x), 0x01010101, ra[0]); ra[1] = __dp4a(static_cast<int>(v.y), 0x01010101, ra[1]);
              ra[2] = __dp4a(static_cast<int>(v.z), 0x01010101, ra[2]); ra[3] = __dp4a(static_cast<int>(v.w), 0x01010101, ra[3]);
            }
            if (two) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const uint4 v = *reinterpret_cast<const uint4*>(slot + (lane + 32) * 128 + (((j + lane) & 7) << 4));
                rb[0] = __dp4a(static_cast<int>(v.x), 0x01010101, rb[0]); rb[1] = __dp4a(static_cast<int>(v.y), 0x01010101, rb[1]);
                rb[2] = __dp4a(static_cast<int>(v.z), 0x01010101, rb[2]); rb[3] = __dp4a(static_cast<int>(v.w), 0x01010101, rb[3]);
              }
            }
            sh->rsum[st][lane] = __int2float_rn((ra[0] + ra[1]) + (ra[2] + ra[3]));
            sh->rsum[st][lane + 32] = __int2float_rn((rb[0] + rb[1]) + (rb[2] + rb[3]));
            sh->tscale[st][0][lane] = cur[0][u] * cur[2][u];
            sh->tscale[st][1][lane] = cur[0][u] * cur[3][u];
            sh->tscale[st][0][lane + 32] = cur[1][u] * cur[2][u];
            sh->tscale[st][1][lane + 32] = cur[1][u] * cur[3][u];
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&sh->x_full[st]);
            if (++st == kTStages) { st = 0; pt ^= 1u; }
          }
        }
      }
    }
  } else if (warp >= kConvWarp0) {
    // ---- converters: packed word -> eight int8 nibbles, written where the tensor core expects them -------------------
    ptx::setmaxnreg_dec<kRegsConv>();
    // Thread (u, c4) of the warp for lane quarter q reads the words w(R, k .. k+3) of packed row R = 8 q + rho(u): eight
    // channels at four k.  A 4 x 4 byte transposition gathers byte j of the four words (nibbles 2j and 2j + 1, i.e. channels
    // 8 R + 2 j and 8 R + 2 j + 1, at four consecutive k): low nibbles are one operand column of half 0, high nibbles of
    // half 1, both in lane u + 8 j.  That is the register layout of tcgen05.st.16x128b (thread: lanes u and u + 8, column
    // c4 of every four), so the operand needs no pass through shared memory: 20 integer instructions per 32 weights.
    // rho pairs rows whose swizzled chunks fall into different bank halves: a quarter-warp reads 128 distinct bytes.
    const int cw = warp - kConvWarp0, q = cw & 3, kh = cw >> 2;    // kh: which 64 of the K block's 128 k
    const int u = lane >> 2, rho = packed_row(u);
    const uint32_t ld_off = (q >> 1) * (kPBytes / 2) + kh * 4096 + ((q & 1) * 8 + rho) * 128;
    const uint32_t col0 = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(kh) * 16u;
    int sp = 0, so = 0;
    uint32_t pp = 0, po = 0;
    bool ok = true;
    for (int t = first; ok && t < total_tiles; t += step) {
      for (int kb = 0; kb < KB; ++kb) {
        if (!warp_wait(&sh->p_full[sp], pp, abort_flag)) { ok = false; break; }
        const uint8_t* src = smem_p + size_t(sp) * kPBytes + ld_off;
        uint32_t o[2][2][8];                                       // [half][lane group of 16][column group, lane + 0 / 8]
#pragma unroll
        for (int i = 0; i < 4; ++i) {                              // 16 k each
          const uint4 w = *reinterpret_cast<const uint4*>(src + (i >> 1) * 2048 + ((((i & 1) * 4 + (lane & 3)) ^ rho) << 4));
          const uint32_t ab = __byte_perm(w.x, w.y, 0x5140), cd = __byte_perm(w.z, w.w, 0x5140);
          const uint32_t ef = __byte_perm(w.x, w.y, 0x7362), gh = __byte_perm(w.z, w.w, 0x7362);
          const uint32_t tb[4] = {__byte_perm(ab, cd, 0x5410), __byte_perm(ab, cd, 0x7632),
                                  __byte_perm(ef, gh, 0x5410), __byte_perm(ef, gh, 0x7632)};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            o[0][j >> 1][2 * i + (j & 1)] = tb[j] & 0x0F0F0F0Fu;
            o[1][j >> 1][2 * i + (j & 1)] = (tb[j] >> 4) & 0x0F0F0F0Fu;
          }
        }
        if (!warp_wait(&sh->op_empty[so], po ^ 1u, abort_flag)) { ok = false; break; }
        if (lane == 0) ptx::mbar_arrive(&sh->p_empty[sp]);         // converged after the wait: every lane has its words
        ptx::tc_fence_after_sync();
        const uint32_t col = col0 + static_cast<uint32_t>(so) * kOpCols;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int g = 0; g < 2; ++g) ptx::tmem_st_16x128b_x4(col + h * (kOpCols / 2) + (static_cast<uint32_t>(g * 16) << 16), o[h][g]);
        ptx::tmem_st_wait();
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sh->op_full[so]);
        if (++sp == kPStages) { sp = 0; pp ^= 1u; }
        if (++so == kOpStages) { so = 0; po ^= 1u; }
      }
    }
  } else {
    // ---- promotion and epilogue: thread = one output channel, registers = tokens -------------------------------------
    ptx::setmaxnreg_inc<kRegsPromo>();
    // TMEM lane u + 8 j of quarter q holds channels c (half 0) and c + 1 (half 1) of the tile: c = 8 (8 q + rho(u)) + 2 j.
    // Quarters 0 and 1 are the tile's first 128-channel block, 2 and 3 its second.
    const int e = warp - kPromoWarp0, q = warp & 3, half = e >> 2, blk = q >> 1;
    const int c = 8 * (8 * q + packed_row(lane & 7)) + 2 * (lane >> 3) + half;
    const uint32_t acc_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + kAccCol + static_cast<uint32_t>(half) * kChunk;
    int as = 0, sr = 0, epi_n = 0;
    uint32_t pacc = 0;
    bool ok = true;
    for (int t = first; ok && t < total_tiles; t += step) {
      const Tile8 tl = decode_tile8(sh, p, t, num_ct);
      int n0, n1;
      half_ch(tl, n0, n1);
      const int ch = blk ? n1 + c - 128 : n0 + c;           // past N: a second block that does not exist
      // K loop and epilogue exist once per number of 16-token blocks, so that the code a tile runs is short and straight
      // (a single version unrolled for 64 tokens spent more time fetching instructions than executing them).
      auto tile_body = [&](auto nblocks) {
      constexpr int kBlocks = decltype(nblocks)::value;
      float acc[kBlocks * 16];
#pragma unroll
      for (int m = 0; m < kBlocks * 16; ++m) acc[m] = 0.f;
      for (int kb = 0; kb < KB; ++kb) {
        // tmem_full alone: the MMAs of this K block were issued after x_full, which follows t_full, so the sums, the
        // scales and the (s4, z4) pairs of this stage are in place (acquire/release chain over the three barriers)
        if (!warp_wait(&sh->tmem_full[as], pacc, abort_flag)) { ok = false; break; }
        ptx::tc_fence_after_sync();
        const uint32_t tcol = acc_base + static_cast<uint32_t>(as) * (2 * kChunk);
        uint32_t d[2][16];                             // the next 16 tokens are in flight while these are worked on
        ptx::tmem_ld16(tcol, d[0]);
        if constexpr (kBlocks > 1) ptx::tmem_ld16(tcol + 16, d[1]);
        const uint32_t zs = sh->sz[sr][c];
        const float s4 = __int2float_rn(static_cast<int8_t>(zs & 0xFFu)), nz = -__int2float_rn(static_cast<int8_t>(zs >> 8));
        const uint64_t s2 = ptx::pack_f32x2(s4, s4), nz2 = ptx::pack_f32x2(nz, nz);
        const ulonglong2* rsp = reinterpret_cast<const ulonglong2*>(sh->rsum[sr]);
        const ulonglong2* tsp = reinterpret_cast<const ulonglong2*>(sh->tscale[sr][blk]);
#pragma unroll
        for (int mb = 0; mb < kBlocks; mb += 2) {
          ptx::tmem_ld_wait16(d[0], d[1]);
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            if (mb + b >= kBlocks) break;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const ulonglong2 r2 = rsp[(mb + b) * 4 + j], t2 = tsp[(mb + b) * 4 + j];
              promote2(acc[(mb + b) * 16 + j * 4], acc[(mb + b) * 16 + j * 4 + 1], d[b][j * 4], d[b][j * 4 + 1], r2.x, nz2, s2, t2.x);
              promote2(acc[(mb + b) * 16 + j * 4 + 2], acc[(mb + b) * 16 + j * 4 + 3], d[b][j * 4 + 2], d[b][j * 4 + 3], r2.y, nz2, s2, t2.y);
            }
            if (mb + b + 2 < kBlocks) ptx::tmem_ld16(tcol + (mb + b + 2) * 16, d[b]);
          }
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) { ptx::mbar_arrive(&sh->tmem_empty[as]); ptx::mbar_arrive(&sh->t_empty[sr]); }
        if (++as == kAccStages) { as = 0; pacc ^= 1u; }
        if (++sr == kTStages) sr = 0;
      }
      if (!ok) return;

      if (!p.fused) {
        if (ch < p.N) {
          uint8_t* dst = static_cast<uint8_t*>(p.c) + static_cast<int64_t>(tl.m0) * p.c_stride + static_cast<int64_t>(ch) * (p.c_dtype == B200MOE_F32 ? 4 : 2);
          if (p.c_dtype == B200MOE_F32) {
#pragma unroll
            for (int m = 0; m < kBlocks * 16; ++m)
              if (m < tl.rows) *reinterpret_cast<float*>(dst + m * p.c_stride) = acc[m];
          } else if (p.c_dtype == B200MOE_BF16) {
#pragma unroll
            for (int m = 0; m < kBlocks * 16; ++m)
              if (m < tl.rows) *reinterpret_cast<__nv_bfloat16*>(dst + m * p.c_stride) = __float2bfloat16_rn(acc[m]);
          } else {
#pragma unroll
            for (int m = 0; m < kBlocks * 16; ++m)
              if (m < tl.rows) *reinterpret_cast<__half*>(dst + m * p.c_stride) = __float2half_rn(acc[m]);
          }
        }
      } else {
        // act(gate) * up with the roundings of the unfused chain (GEMM output, activation and product each rounded
        // to bf16; moe/group_gemm_kernel.py:120-235), then the int8 1x128 quantizer of
        // quantization/w4a8_kernel.py:145-168: s = amax / 127, y = floor(h / s + 0.5), s stored after an f16 rounding.
        // Gate and up (held by different warps) go through a [token][channel] bf16 stage in shared memory (exact: they
        // are bf16 values); a warp then owns whole tokens: maximum by shuffles, four channels per lane, one 128-byte row
        // per store.
        const uint32_t par = static_cast<uint32_t>(epi_n & 1);
        if (!warp_wait(&sh->stage_free, par ^ 1u, abort_flag)) { ok = false; return; }     // previous tile's readers are done
#pragma unroll
        for (int m = 0; m < kBlocks * 16; ++m) sh->stage[m][c] = __float2bfloat16_rn(acc[m]);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sh->stage_full);
        if (!warp_wait(&sh->stage_full, par, abort_flag)) { ok = false; return; }
        ++epi_n;
        for (int m = e; m < tl.rows; m += kPromoWarps) emit_row(sh, p, tl, m);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sh->stage_free);
      }
      };
      switch (tl.tn >> 4) {
        case 1: tile_body(std::integral_constant<int, 1>{}); break;
        case 2: tile_body(std::integral_constant<int, 2>{}); break;
        case 3: tile_body(std::integral_constant<int, 3>{}); break;
        default: tile_body(std::integral_constant<int, 4>{}); break;
      }
    }
  }

  // ---- teardown ------------------------------------------------------------------------------------------
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc<1>(tmem_base, kTmemCols);
  if (threadIdx.x == 0 && sh->abort_flag && p.status) *p.status = B200MOE_DEVICE_TIMEOUT;
}

}  // namespace w4
}  // namespace b200moe

using namespace b200moe;

extern "C" int b200moe_grouped_gemm_w4a8(const void* a, int64_t a_row_stride_bytes, const float* a_s,
                                         int64_t a_s_row_stride, const void* b_packed, const void* s4z4_t,
                                         const float* b_s, void* c, int c_dtype, int64_t c_row_stride_bytes,
                                         float* c_s, int64_t c_s_row_stride, int64_t M_total, int64_t N, int64_t K,
                                         int num_groups, int num_weights, const int64_t* seg_indptr,
                                         const int64_t* weight_indices, int epilogue, int32_t* status_word,
                                         void* stream) {
  B200MOE_REQUIRE(a && a_s && b_packed && s4z4_t && b_s && c && seg_indptr, B200MOE_BAD_ARG, "grouped_gemm_w4a8: null pointer");
  B200MOE_REQUIRE(epilogue == 0 || epilogue == 1 || epilogue == 4, B200MOE_BAD_ARG, "grouped_gemm_w4a8: epilogue %d", epilogue);
  B200MOE_REQUIRE(M_total >= 0 && M_total < (int64_t(1) << 31) && N > 0 && K > 0 && K % 128 == 0 && N % 128 == 0,
                  B200MOE_BAD_SHAPE, "grouped_gemm_w4a8: M=%lld N=%lld K=%lld (N and K must be multiples of 128)",
                  (long long)M_total, (long long)N, (long long)K);
  B200MOE_REQUIRE(num_groups >= 1 && num_groups <= w4::kMaxGroups && num_weights >= 1 &&
                  static_cast<int64_t>(num_weights) * N < (int64_t(1) << 31), B200MOE_BAD_SHAPE,
                  "grouped_gemm_w4a8: num_groups=%d (max %d) num_weights=%d", num_groups, w4::kMaxGroups, num_weights);
  B200MOE_REQUIRE(aligned(a, 16) && aligned(b_packed, 16) && aligned(s4z4_t, 16) && aligned(c, 16) &&
                  a_row_stride_bytes % 16 == 0 && a_row_stride_bytes >= K && c_row_stride_bytes % 16 == 0,
                  B200MOE_BAD_ALIGN, "grouped_gemm_w4a8: pointers and row strides must be 16-byte aligned");
  B200MOE_REQUIRE(a_s_row_stride >= K / 128, B200MOE_BAD_ARG, "grouped_gemm_w4a8: a_s row stride too small");
  if (epilogue != 0) {
    B200MOE_REQUIRE(N % 256 == 0, B200MOE_BAD_SHAPE, "grouped_gemm_w4a8: the fused epilogue needs N %% 256 == 0, got %lld", (long long)N);
    B200MOE_REQUIRE(c_dtype == B200MOE_I8 && c_s && c_row_stride_bytes >= N / 2 && c_s_row_stride >= N / 256,
                    B200MOE_BAD_ARG, "grouped_gemm_w4a8: the fused epilogue writes int8 rows and f32 scales");
  } else {
    B200MOE_REQUIRE(c_dtype == B200MOE_F32 || c_dtype == B200MOE_F16 || c_dtype == B200MOE_BF16, B200MOE_BAD_DTYPE,
                    "grouped_gemm_w4a8: c dtype %d", c_dtype);
    B200MOE_REQUIRE(c_row_stride_bytes >= N * (c_dtype == B200MOE_F32 ? 4 : 2), B200MOE_BAD_ARG, "grouped_gemm_w4a8: c row stride too small");
  }
  if (M_total == 0) return B200MOE_OK;
  int sms = 0;
  if (int rc = require_sm100(&sms)) return rc;
  w4::RowMaps ma;
  CUtensorMap mp;
  for (int i = 0; i < 3; ++i)
    if (int rc = cached_tensor_map_u8(&ma.m[i], a, static_cast<uint64_t>(M_total), static_cast<uint64_t>(K),
                                      static_cast<uint64_t>(a_row_stride_bytes), 16u << i)) return rc;
  ma.m[3] = ma.m[2];
  if (int rc = make_tensor_map_i32_kgroups(&mp, b_packed, static_cast<uint64_t>(num_weights) * (N / 8), static_cast<uint64_t>(K), 16)) return rc;
  w4::Params8 p{a_s, a_s_row_stride, b_s, static_cast<const uint16_t*>(s4z4_t), c, c_row_stride_bytes, c_s, c_s_row_stride,
                seg_indptr, weight_indices, M_total, static_cast<int>(N), static_cast<int>(K), num_groups, c_dtype,
                epilogue != 0 ? 1 : 0, epilogue == 4 ? 1 : 0, status_word};
  if (int rc = set_dynamic_smem(reinterpret_cast<const void*>(w4::gemm_w4a8_kernel), w4::kSmem8)) return rc;
  // a plain launch: as dependent launches these long kernels gained nothing (DeepSeek-V3 layer of 64 tokens 1273 us either way, of
  // 3000 tokens 4585 us plain, 4637 dependent; two runs of one side differ by 0.5 %)
  w4::gemm_w4a8_kernel<<<sms, w4::kThreads8, w4::kSmem8, as_stream(stream)>>>(ma, mp, p);
  return check_launch("gemm_w4a8_kernel");
}
