// Grouped w4a16 GEMM (asymmetric group-128 int4 weights, w = bf16((q - zero) * scale), bf16 activations, f32 accumulation) with
// the dequantization fused into the operand path (no expanded copy of the weights).
//
// What bounds it: the conversion of every packed weight to bf16 by the CUDA cores, once per chunk of tokens, then the packed
// bytes themselves.  The weights are the M = 128 side of the MMA and their operand lives in TENSOR MEMORY: lane = output
// channel, column = two consecutive k.  A converter thread owns one channel, reads its packed words (eight consecutive k each,
// quantization/bitpack.py:38-67) from the TMA ring and stores bf16 pairs with tcgen05.st; the converted weights never touch
// shared memory, whose traffic (write the 32 KB tile, read it and a 128-row token tile for the MMA) bounded a version with
// the tokens on the M side.  The tokens are the N = 16..CHUNK columns, so few rows cost little tensor-core time.
//
// Measured on 8 experts of a Mixtral layer (gate/up N 28672 K 4096, then down N 4096 K 14336; us; tokens on the M side and
// weights through shared memory -> here): 1-16 rows per expert 436 + 219 -> 186 + 98, 64 rows 440 + 221 -> 223 + 101,
// 128 rows 451 + 225 -> 291 + 120, 256 rows 821 + 438 -> 514 + 222.  The roles that are one thread are entered through
// elect.sync: under `lane == 0` every tcgen05 instruction took about 90 cycles to issue, 750 cycles for the MMAs of 64 k
// instead of 150.  Even so the MMA thread's barriers counted: one hand-over per 128 k instead of two 205 + 108 -> 186 + 98.
//
// One persistent CTA per SM, 768 threads:
//   warp 0       TMA producer of the packed words: two boxes of 128 channels x 128 B (256 k) and their (scale, zero)
//                pairs as bulk copies, 4 slots of 34 KB
//   warp 2       TMA producer of the token rows: two boxes of 16/32/64/128 rows x 64 k, 64 KB ring
//   warps 8-23   converters: warp w serves TMEM lanes 32 (w % 4).. of channel half (w / 4) % 2 and every other K block of 128
//   warp 1       owns TMEM: 2 operand stages of 128 columns, 256 columns of accumulators; per K block 2 x 8
//                tcgen05.mma.kind::f16 (M128, N = tokens, K16); the whole K loop accumulates in TMEM
//   warps 4-7    tile epilogue (plain, or act(gate) * up); with CHUNK = 64 it overlaps the next tile
//
// Every wait is a bounded mbarrier wait; on expiry the kernel drains its copies, frees TMEM, writes
// B200MOE_DEVICE_TIMEOUT to the status word and returns.
#include <cuda.h>

#include "common.cuh"
#include "epilogue.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"
#include "w4_common.cuh"

namespace b200moe {
namespace w4a16 {

constexpr int kWStages = 4, kOpStages = 2;
constexpr uint32_t kWBytes = 2 * 128 * 128;            // two halves of 128 channels x 32 words (256 k)
constexpr uint32_t kPairBytes = 128 * 4;               // (scale, zero) of one half and one 128-k group
constexpr uint32_t kWSlot = kWBytes + 4 * kPairBytes;  // [group][half][128] pairs behind the words
constexpr uint32_t kTRing = 65536;                     // token ring: 4 slots of 64 rows or 2 of 128 rows, two boxes of 64 k each
constexpr int kMaxTStages = 4;
constexpr uint32_t kOpCols = 128;                      // operand stage: [64-k block of the pair][half][32 columns]
constexpr int kThreads = 768, kEpiWarp0 = 4, kEpiWarps = 4, kConvWarp0 = 8, kConvWarps = 16;
constexpr uint32_t kAccCol = 256;                      // first accumulator column
static_assert(kWSlot % 1024 == 0, "the 128-byte swizzle needs 1 KB aligned slots");

struct Tail {
  uint64_t w_full[kWStages], w_empty[kWStages];
  uint64_t t_full[kMaxTStages], t_empty[kMaxTStages];
  uint64_t op_full[kOpStages], op_empty[kOpStages];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int32_t seg[w4::kMaxGroups + 1];
  int32_t pref[w4::kMaxGroups + 1];                    // exclusive prefix of token chunks per group
};
constexpr size_t kSmem = 1024 + size_t(kWStages) * kWSlot + kTRing + sizeof(Tail);
static_assert(kSmem <= 232448, "shared memory of one CTA");

struct Params {
  const uint32_t* sz_t;           // [W, K/128, N]: (scale, zero) bf16 pairs (scale in the low half)
  void* c; int64_t c_stride;      // bytes
  const int64_t* seg; const int64_t* widx;
  int N, K, num_groups, c_dtype, fused, act;
  int32_t* status;
};

struct Tile { int m0, rows, tn, expert, ct; };

template <int CHUNK>
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
  tl.m0 = sh->seg[lo] + (rem - tl.ct * chunks) * CHUNK;
  tl.rows = min(CHUNK, sh->seg[lo + 1] - tl.m0);
  tl.tn = (tl.rows + 15) & ~15;
  tl.expert = p.widx ? static_cast<int>(p.widx[lo]) : lo;
  return tl;
}

__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag));
}

__device__ __forceinline__ uint32_t bf2_bits(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ __nv_bfloat162 bits_bf2(uint32_t v) { return *reinterpret_cast<const __nv_bfloat162*>(&v); }

// One packed word (nibble i = k 8c + i) -> eight bf16 values (q - zero) * scale as four bf16x2 registers in k order.
// 0x4300 | q is the bf16 number 128 + q; the two subtractions are exact and the product is rounded once, which is
// the f32 evaluation of (q - zero) * scale rounded to bf16.
__device__ __forceinline__ uint4 dequant_word_bf16(uint32_t w, uint32_t scale_zero) {
  const __nv_bfloat162 sc = __bfloat162bfloat162(__ushort_as_bfloat16(static_cast<unsigned short>(scale_zero & 0xFFFFu)));
  const __nv_bfloat162 zp = __bfloat162bfloat162(__ushort_as_bfloat16(static_cast<unsigned short>(scale_zero >> 16)));
  const __nv_bfloat162 c128 = __bfloat162bfloat162(__ushort_as_bfloat16(0x4300));
  uint32_t pr[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) pr[j] = ((w >> (4 * j)) & 0x000F000Fu) | 0x43004300u;     // (nibble j, nibble j + 4)
  const uint32_t o[4] = {__byte_perm(pr[0], pr[1], 0x5410), __byte_perm(pr[2], pr[3], 0x5410),
                         __byte_perm(pr[0], pr[1], 0x7632), __byte_perm(pr[2], pr[3], 0x7632)};
  uint32_t r[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&o[j]);
    v = __hmul2(__hsub2(__hsub2(v, c128), zp), sc);
    r[j] = *reinterpret_cast<const uint32_t*>(&v);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}

// One channel's (scale, zero) of a 128-k group, prepared for convert_word: v = (x - c) * s on bf16 pairs, where x holds
// 128 + q of an even k and 128 + 8 q of the odd k after it.
struct Affine { uint32_t c, s; bool whole; };
__device__ __forceinline__ Affine make_affine(uint32_t scale_zero) {
  const uint32_t sb = scale_zero & 0xFFFFu;
  const float z = __uint_as_float(scale_zero & 0xFFFF0000u), s = __uint_as_float(sb << 16);
  Affine a;
  // 128 + z and 128 + 8 z are bf16 numbers when z is a whole number of 0..15, and s / 8 is exact unless it underflows:
  // then the one subtraction gives q - z (8 (q - z)) exactly and the product rounds the same real number as
  // (q - z) * s.  Zero points or scales outside take the general form.
  a.whole = z >= 0.f && z <= 15.f && z == (z + 12582912.f) - 12582912.f && ((sb & 0x7F80u) >= (4u << 7) || (sb & 0x7FFFu) == 0u);
  a.c = bf2_bits(__floats2bfloat162_rn(128.f + z, 128.f + 8.f * z));
  a.s = bf2_bits(__floats2bfloat162_rn(s, s * 0.125f));
  return a;
}
// Eight nibbles (nibble i = k 8c + i) -> four bf16 pairs in k order: 17 instructions.
__device__ __forceinline__ void convert_word(uint32_t w, const Affine& a, uint32_t* r) {
  const uint32_t w1 = w >> 1;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    // byte b holds nibbles 2b (bits 0-3) and 2b + 1 (bits 3-6 after the shift): 0x4300 | q is 128 + q in bf16
    const uint32_t x = (__byte_perm(w, w1, b | (b << 4) | ((4 + b) << 8) | ((4 + b) << 12)) & 0x0078000Fu) | 0x43004300u;
    r[b] = bf2_bits(__hmul2(__hsub2(bits_bf2(x), bits_bf2(a.c)), bits_bf2(a.s)));
  }
}

template <int CHUNK>
__global__ void __launch_bounds__(kThreads, 1)
gemm_w4a16_kernel(const __grid_constant__ w4::RowMaps tmap_a, const __grid_constant__ CUtensorMap tmap_p,
                  const __grid_constant__ Params p) {
  constexpr int kTStages = static_cast<int>(kTRing / (CHUNK * 256));
  constexpr int kAccStages = 128 / CHUNK;              // CHUNK = 64: two, CHUNK = 128: one
  static_assert(kTStages <= kMaxTStages && kAccStages >= 1, "");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_t = smem + size_t(kWStages) * kWSlot;
  Tail* sh = reinterpret_cast<Tail*>(smem_t + kTRing);
  volatile int* abort_flag = &sh->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KG = p.K / 128;                            // K blocks: one scale group, two 64-k boxes of the swizzle
  const int KW = (KG + 1) / 2;                         // 256-k slots of packed words, the last one maybe half
  const int num_ct = p.fused ? p.N / 256 : (p.N + 255) / 256;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kWStages; ++s) { ptx::mbar_init(&sh->w_full[s], 1); ptx::mbar_init(&sh->w_empty[s], kConvWarps); }
    for (int s = 0; s < kTStages; ++s) { ptx::mbar_init(&sh->t_full[s], 1); ptx::mbar_init(&sh->t_empty[s], 1); }
    for (int s = 0; s < kOpStages; ++s) { ptx::mbar_init(&sh->op_full[s], kConvWarps / 2); ptx::mbar_init(&sh->op_empty[s], 1); }
    for (int s = 0; s < kAccStages; ++s) { ptx::mbar_init(&sh->acc_full[s], 1); ptx::mbar_init(&sh->acc_empty[s], kEpiWarps); }
    sh->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
#pragma unroll
    for (int i = 0; i < 4; ++i) ptx::prefetch_tensormap(&tmap_a.m[i]);
    ptx::prefetch_tensormap(&tmap_p);
  }
  if (warp == 1) {
    ptx::tmem_alloc<1>(&sh->tmem_base, w4::kTmemCols);
    ptx::tmem_relinquish<1>();
  }
  // the setup above overlaps the tail of the kernel before; from here on its results are read
  wait_for_predecessors();
  for (int g = threadIdx.x; g <= p.num_groups; g += kThreads) sh->seg[g] = static_cast<int32_t>(p.seg[g]);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  if (warp == 3) {
    int run = 0;
    for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
      const int g = g0 + lane;
      int v = 0;
      if (g < p.num_groups) { const int m = sh->seg[g + 1] - sh->seg[g]; v = m > 0 ? (m + CHUNK - 1) / CHUNK : 0; }
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
  const int total = sh->pref[p.num_groups] * num_ct, first = static_cast<int>(blockIdx.x), step = static_cast<int>(gridDim.x);
  // first output channel of the tile's two halves (within the expert's N channels)
  auto half_ch = [&](const Tile& tl, int& n0, int& n1) {
    n0 = p.fused ? tl.ct * 128 : tl.ct * 256;
    n1 = p.fused ? p.N / 2 + tl.ct * 128 : n0 + 128;
  };

  if (warp == 0 && ptx::elect_one()) {
    // ---- packed words and their (scale, zero) pairs ----------------------------------------------------------------
    int stage = 0; uint32_t phase = 0;
    w4::Armed armed;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = decode<CHUNK>(sh, p, t, num_ct);
      int n0, n1;
      half_ch(tl, n0, n1);
      const bool second = n1 < p.N;
      const int row0 = tl.expert * p.N + n0, row1 = tl.expert * p.N + n1;
      const uint32_t* sz = p.sz_t + static_cast<int64_t>(tl.expert) * (p.K / 128) * p.N;
      for (int kw = 0; kw < KW; ++kw) {
        if (!ptx::mbar_wait(&sh->w_empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
        uint8_t* sw = smem + size_t(stage) * kWSlot;
        const bool two = kw * 2 + 1 < KG;              // the slot's second 128-k group exists
        ptx::mbar_arrive_expect_tx(&sh->w_full[stage], (kWBytes / 2 + kPairBytes * (two ? 2u : 1u)) * (second ? 2u : 1u));
        armed.arm(stage, phase);
        ptx::tma_load_2d(sw, &tmap_p, &sh->w_full[stage], kw * 32, row0);          // words past K: zero fill
        const uint32_t* szk = sz + static_cast<int64_t>(kw) * 2 * p.N;
        ptx::bulk_load(sw + kWBytes, szk + n0, kPairBytes, &sh->w_full[stage]);
        if (two) ptx::bulk_load(sw + kWBytes + 2 * kPairBytes, szk + p.N + n0, kPairBytes, &sh->w_full[stage]);
        if (second) {
          ptx::tma_load_2d(sw + kWBytes / 2, &tmap_p, &sh->w_full[stage], kw * 32, row1);
          ptx::bulk_load(sw + kWBytes + kPairBytes, szk + n1, kPairBytes, &sh->w_full[stage]);
          if (two) ptx::bulk_load(sw + kWBytes + 3 * kPairBytes, szk + p.N + n1, kPairBytes, &sh->w_full[stage]);
        }
        if (++stage == kWStages) { stage = 0; phase ^= 1u; }
      }
    }
    if (!ok) armed.drain(sh->w_full, kWStages);
  } else if (warp == 2 && ptx::elect_one()) {
    // ---- token rows ------------------------------------------------------------------------------------------------
    int stage = 0; uint32_t phase = 0;
    w4::Armed armed;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = decode<CHUNK>(sh, p, t, num_ct);
      const int sel = tl.tn <= 16 ? 0 : (tl.tn <= 32 ? 1 : (tl.tn <= 64 ? 2 : 3));
      for (int kg = 0; kg < KG; ++kg) {
        if (!ptx::mbar_wait(&sh->t_empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
        ptx::mbar_arrive_expect_tx(&sh->t_full[stage], (16u << sel) * 256u);
        armed.arm(stage, phase);
        uint8_t* slot = smem_t + size_t(stage) * (CHUNK * 256);
        ptx::tma_load_2d(slot, &tmap_a.m[sel], &sh->t_full[stage], kg * 256, tl.m0);
        ptx::tma_load_2d(slot + CHUNK * 128, &tmap_a.m[sel], &sh->t_full[stage], kg * 256 + 128, tl.m0);
        if (++stage == kTStages) { stage = 0; phase ^= 1u; }
      }
    }
    if (!ok) armed.drain(sh->t_full, kTStages);
  } else if (warp == 1 && ptx::elect_one()) {
    // ---- MMA issuer: channels (tensor memory) are the M = 128 rows, tokens (shared memory) the N columns -----------
    int so = 0, st = 0, as = 0;
    uint32_t po = 0, pt = 0, pacc = 0;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = decode<CHUNK>(sh, p, t, num_ct);
      const uint32_t idesc = ptx::umma_idesc(1, 1, 1, 128, static_cast<uint32_t>(tl.tn));    // D f32, A and B bf16
      if (!ptx::mbar_wait(&sh->acc_empty[as], pacc ^ 1u, abort_flag)) break;     // the stage's previous tile has been read
      const uint32_t d = tmem_base + kAccCol + static_cast<uint32_t>(as) * (2 * CHUNK);
      for (int kg = 0; kg < KG; ++kg) {
        if (!ptx::mbar_wait(&sh->t_full[st], pt, abort_flag) || !ptx::mbar_wait(&sh->op_full[so], po, abort_flag)) { ok = false; break; }
        ptx::tc_fence_after_sync();
        const uint32_t a = tmem_base + static_cast<uint32_t>(so) * kOpCols;
        const uint64_t tdesc = ptx::umma_desc_sw128(ptx::smem_u32(smem_t + size_t(st) * (CHUNK * 256)));
#pragma unroll
        for (int k = 0; k < 8; ++k) {      // halves alternate: an instruction does not wait for the one that feeds its accumulator
          const uint64_t td = tdesc + (k >> 2) * (CHUNK * 128 >> 4) + 2 * (k & 3);
          const uint32_t ak = a + 64u * (k >> 2) + 8u * (k & 3), more = (kg > 0 || k > 0) ? 1u : 0u;
          ptx::umma_f16_ts(d, ak, td, idesc, more);
          ptx::umma_f16_ts(d + CHUNK, ak + 32u, td, idesc, more);
        }
        ptx::umma_commit(&sh->op_empty[so]);
        ptx::umma_commit(&sh->t_empty[st]);
        if (++so == kOpStages) { so = 0; po ^= 1u; }
        if (++st == kTStages) { st = 0; pt ^= 1u; }
      }
      if (!ok) break;
      ptx::umma_commit(&sh->acc_full[as]);               // the tile's accumulators are complete
      if (++as == kAccStages) { as = 0; pacc ^= 1u; }
    }
  } else if (warp >= kConvWarp0) {
    // ---- converters: thread = output channel, one K block (16 packed words) at a time; the two groups take turns ------
    const int cw = warp - kConvWarp0;
    const int q = cw & 3, half = (cw >> 2) & 1, par = cw >> 3;   // kConvWarp0 % 4 == 0: TMEM lane quarter = warp % 4
    const int row = q * 32 + lane;                                // channel within the half = TMEM lane
    const uint8_t* my_w = smem + half * (kWBytes / 2) + row * 128;
    const uint8_t* my_sz = smem + kWBytes + half * kPairBytes + row * 4;
    // operand stage = group: the K blocks of all tiles in turn, stage 0 and stage 1 alternating
    const uint32_t my_t = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(par) * kOpCols + static_cast<uint32_t>(half) * 32u;
    int sw = 0, turn = 0;
    uint32_t pw = 0, po = 0;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      for (int kw = 0; ok && kw < KW; ++kw) {
        if (!warp_wait(&sh->w_full[sw], pw, abort_flag)) { ok = false; break; }
        const int blocks = min(2, KG - kw * 2);
        const int mine = (turn ^ par) & 1;                        // this group's K block of the slot
        turn += blocks;
        if (mine < blocks) {
          const uint8_t* src = my_w + size_t(sw) * kWSlot;
          const uint32_t sz = *reinterpret_cast<const uint32_t*>(my_sz + size_t(sw) * kWSlot + mine * (2 * kPairBytes));
          const Affine a = make_affine(sz);
          const bool whole = __all_sync(0xffffffffu, a.whole);
#pragma unroll 1
          for (int s = 0; s < 2; ++s) {                           // 64 k each
            const int ch = mine * 4 + s * 2;
            const uint4 wa = *reinterpret_cast<const uint4*>(src + ((ch ^ (row & 7)) << 4));
            const uint4 wb = *reinterpret_cast<const uint4*>(src + (((ch + 1) ^ (row & 7)) << 4));
            const uint32_t wd[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
            uint32_t r[32];
            if (whole) {
#pragma unroll
              for (int i = 0; i < 8; ++i) convert_word(wd[i], a, r + 4 * i);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint4 v = dequant_word_bf16(wd[i], sz);
                r[4 * i] = v.x; r[4 * i + 1] = v.y; r[4 * i + 2] = v.z; r[4 * i + 3] = v.w;
              }
            }
            if (s == 0) {
              if (!warp_wait(&sh->op_empty[par], po ^ 1u, abort_flag)) { ok = false; break; }
              ptx::tc_fence_after_sync();
            }
            ptx::tmem_st32(my_t + static_cast<uint32_t>(s) * 64u, r);
          }
          if (!ok) break;
          ptx::tmem_st_wait();
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&sh->op_full[par]);
          po ^= 1u;
        }
        if (lane == 0) ptx::mbar_arrive(&sh->w_empty[sw]);        // converged: every lane has read its words
        if (++sw == kWStages) { sw = 0; pw ^= 1u; }
      }
    }
  } else if (warp >= kEpiWarp0) {
    // ---- epilogue: thread = output channel (one of each half) --------------------------------------------------------
    const int q = warp & 3, c = q * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    int as = 0;
    uint32_t pacc = 0;
    for (int t = first; t < total; t += step) {
      const Tile tl = decode<CHUNK>(sh, p, t, num_ct);
      int n0, n1;
      half_ch(tl, n0, n1);
      const bool second = n1 < p.N;
      if (!warp_wait(&sh->acc_full[as], pacc, abort_flag)) break;
      ptx::tc_fence_after_sync();
      const uint32_t tcol = tmem_base + lane_base + kAccCol + static_cast<uint32_t>(as) * (2 * CHUNK);
      uint8_t* out = static_cast<uint8_t*>(p.c) + static_cast<int64_t>(tl.m0) * p.c_stride;
#pragma unroll 1
      for (int mb = 0; mb < tl.tn; mb += 16) {
        uint32_t d0[16], d1[16];
        ptx::tmem_ld16(tcol + mb, d0);
        ptx::tmem_ld16(tcol + CHUNK + mb, d1);
        ptx::tmem_ld_wait16(d0, d1);
#pragma unroll
        for (int m = 0; m < 16; ++m) {
          if (mb + m >= tl.rows) break;
          const float v0 = __uint_as_float(d0[m]), v1 = __uint_as_float(d1[m]);
          uint8_t* dst = out + static_cast<int64_t>(mb + m) * p.c_stride;
          if (p.fused) {
            reinterpret_cast<__nv_bfloat16*>(dst)[tl.ct * 128 + c] = __float2bfloat16_rn(bf16r(gate_act(bf16r(v0), p.act)) * bf16r(v1));
          } else if (p.c_dtype == B200MOE_F32) {
            reinterpret_cast<float*>(dst)[n0 + c] = v0;
            if (second) reinterpret_cast<float*>(dst)[n1 + c] = v1;
          } else if (p.c_dtype == B200MOE_BF16) {
            reinterpret_cast<__nv_bfloat16*>(dst)[n0 + c] = __float2bfloat16_rn(v0);
            if (second) reinterpret_cast<__nv_bfloat16*>(dst)[n1 + c] = __float2bfloat16_rn(v1);
          } else {
            reinterpret_cast<__half*>(dst)[n0 + c] = __float2half_rn(v0);
            if (second) reinterpret_cast<__half*>(dst)[n1 + c] = __float2half_rn(v1);
          }
        }
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh->acc_empty[as]);
      if (++as == kAccStages) { as = 0; pacc ^= 1u; }
    }
  }

  // ---- teardown ------------------------------------------------------------------------------------------------
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) ptx::tmem_dealloc<1>(tmem_base, w4::kTmemCols);
  if (threadIdx.x == 0 && sh->abort_flag && p.status) *p.status = B200MOE_DEVICE_TIMEOUT;
}

// Average rows per group above which a tile takes 128 tokens (one set of accumulators) instead of 64 (two sets, the epilogue
// overlaps).  Gate/up above, us: 64 rows per group 213 with chunks of 64, 223 with chunks of 128; 96 rows 263 with chunks of
// 128, where two chunks of 64 would be about 2 x 200.  Groups are ragged, so the line is below 64: from about 48 on average
// some need a second chunk of 64.
constexpr int kWideChunkRows = 48;

template <int CHUNK>
static int launch_chunk(const w4::RowMaps& ma, const CUtensorMap& mp, const Params& p, int sms, cudaStream_t st) {
  if (int rc = set_dynamic_smem(reinterpret_cast<const void*>(gemm_w4a16_kernel<CHUNK>), kSmem)) return rc;
  return launch_dependent("gemm_w4a16_kernel", gemm_w4a16_kernel<CHUNK>, dim3(static_cast<unsigned>(sms)), kThreads, kSmem, st, ma, mp, p);
}

static int launch(const void* a, int64_t a_stride, const void* b_packed, const void* scale_zero_t, void* c, int c_dtype,
                  int64_t c_stride, int64_t M_total, int64_t N, int64_t K, int num_groups, int num_weights, const int64_t* seg,
                  const int64_t* widx, int fused, int act, int32_t* status, cudaStream_t st) {
  int sms = 0;
  if (int rc = require_sm100(&sms)) return rc;
  w4::RowMaps ma;
  CUtensorMap mp;
  for (int i = 0; i < 4; ++i)
    if (int rc = cached_tensor_map_u8(&ma.m[i], a, static_cast<uint64_t>(M_total), static_cast<uint64_t>(2 * K),
                                      static_cast<uint64_t>(a_stride), 16u << i)) return rc;
  if (int rc = make_tensor_map_i32_plain(&mp, b_packed, static_cast<uint64_t>(num_weights) * N, static_cast<uint64_t>(K / 8),
                                         static_cast<uint64_t>(K / 8) * 4, 32, 128, true)) return rc;
  const Params p{static_cast<const uint32_t*>(scale_zero_t), c, c_stride, seg, widx, static_cast<int>(N), static_cast<int>(K),
                 num_groups, c_dtype, fused, act, status};
  return M_total <= kWideChunkRows * static_cast<int64_t>(num_groups) ? launch_chunk<64>(ma, mp, p, sms, st)
                                                                      : launch_chunk<128>(ma, mp, p, sms, st);
}

}  // namespace w4a16
}  // namespace b200moe

using namespace b200moe;

extern "C" int b200moe_grouped_gemm_w4a16(const void* a, int64_t a_row_stride_bytes, const void* b_packed,
                                          const void* scale_zero_t, void* c, int c_dtype, int64_t c_row_stride_bytes,
                                          int64_t M_total, int64_t N, int64_t K, int num_groups, int num_weights,
                                          const int64_t* seg_indptr, const int64_t* weight_indices, int epilogue,
                                          int32_t* status_word, void* stream) {
  B200MOE_REQUIRE(a && b_packed && scale_zero_t && c && seg_indptr, B200MOE_BAD_ARG, "grouped_gemm_w4a16: null pointer");
  B200MOE_REQUIRE(epilogue == 0 || epilogue == 2 || epilogue == 5, B200MOE_BAD_ARG,
                  "grouped_gemm_w4a16: epilogue %d (0 plain, 2 SiLU*up, 5 GELU*up)", epilogue);
  B200MOE_REQUIRE(M_total >= 0 && M_total < (int64_t(1) << 31) && N > 0 && K > 0 && K % 128 == 0 && N % 128 == 0,
                  B200MOE_BAD_SHAPE, "grouped_gemm_w4a16: M=%lld N=%lld K=%lld (N and K must be multiples of 128)",
                  (long long)M_total, (long long)N, (long long)K);
  B200MOE_REQUIRE(num_groups >= 1 && num_groups <= w4::kMaxGroups && num_weights >= 1 &&
                  static_cast<int64_t>(num_weights) * N < (int64_t(1) << 31), B200MOE_BAD_SHAPE,
                  "grouped_gemm_w4a16: num_groups=%d (max %d) num_weights=%d", num_groups, w4::kMaxGroups, num_weights);
  B200MOE_REQUIRE(aligned(a, 16) && aligned(b_packed, 16) && aligned(scale_zero_t, 16) && aligned(c, 16) &&
                  a_row_stride_bytes % 16 == 0 && a_row_stride_bytes >= 2 * K && c_row_stride_bytes % 16 == 0,
                  B200MOE_BAD_ALIGN, "grouped_gemm_w4a16: pointers and row strides must be 16-byte aligned");
  if (epilogue != 0) {
    B200MOE_REQUIRE(N % 256 == 0 && c_dtype == B200MOE_BF16 && c_row_stride_bytes >= N, B200MOE_BAD_ARG,
                    "grouped_gemm_w4a16: the fused epilogue needs N %% 256 == 0 and a bf16 [M, N/2] output");
  } else {
    B200MOE_REQUIRE(c_dtype == B200MOE_F32 || c_dtype == B200MOE_F16 || c_dtype == B200MOE_BF16, B200MOE_BAD_DTYPE,
                    "grouped_gemm_w4a16: c dtype %d", c_dtype);
    B200MOE_REQUIRE(c_row_stride_bytes >= N * (c_dtype == B200MOE_F32 ? 4 : 2), B200MOE_BAD_ARG, "grouped_gemm_w4a16: c row stride too small");
  }
  if (M_total == 0) return B200MOE_OK;
  return w4a16::launch(a, a_row_stride_bytes, b_packed, scale_zero_t, c, c_dtype, c_row_stride_bytes, M_total, N, K, num_groups,
                       num_weights, seg_indptr, weight_indices, epilogue != 0 ? 1 : 0, epilogue == 5 ? 1 : 0, status_word,
                       as_stream(stream));
}
