// int4 weight formats: expansion to the tensor-core operand types.
//
//   two-level int4 (quantization/w4a8_kernel.py:44-101, 196-309): packed int32 [N/8, K] (8 output
//   channels per word, quantization/bitpack.py:9-36), s4/z4 int8 [N, K/128]:
//       w8[n,k] = int8( (q[n,k] - z4[n,k/128]) * s4[n,k/128] )         (int8 wrap as the reference)
//   asymmetric group-128 int4 (extension of fast_dequant/simple_marlin/utils.py:98-136): packed
//   int32 [N, K/8] (8 consecutive k per word, quantization/bitpack.py:38-67), scale/zero bf16
//   [N, K/128]:  w[n,k] = bf16( (q - zero) * scale )
// Both are HBM-bound one-pass kernels over a stack of W matrices.
#include "common.cuh"
#include "marlin_perm.cuh"

namespace b200moe {

// f16 scales that a product wants as f32, turned on the way by the threads of the expansion.
struct ScaleCasts { const __half* src[2]; float* dst[2]; int64_t n[2]; };

// One warp: one packed row (8 channels) and one 128-k group, a lane four consecutive k -> 8 rows x 4 int8.  The int8 wrap makes
// it arithmetic modulo 256: two nibbles in the halves of a register times the scale's byte, plus the byte of -z * s, are one
// multiply-add (at most 15 * 255 + 255, no carry into the upper half).  The channels' scales and zero points are read once per
// warp, by its first lanes.  4096 x 7168 (15 MB in, 29 MB out): 16.9 us with integer arithmetic per nibble, 9.1 us here.
template <typename Index>
__global__ void __launch_bounds__(256) w4a8_expand_kernel(const uint32_t* __restrict__ packed, const int8_t* __restrict__ s4,
                                                          const int8_t* __restrict__ z4, int8_t* __restrict__ out,
                                                          int64_t rows8, int64_t K, const ScaleCasts casts) {
#pragma unroll
  for (int v = 0; v < 2; ++v)
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < casts.n[v];
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) casts.dst[v][i] = __half2float(casts.src[v][i]);
  const Index kg = static_cast<Index>(K / 128), total = static_cast<Index>(rows8) * kg;
  const int lane = threadIdx.x & 31;
  for (Index i = static_cast<Index>(blockIdx.x) * 8 + (threadIdx.x >> 5); i < total; i += static_cast<Index>(gridDim.x) * 8) {
    const Index r = i / kg, g = i - r * kg;
    const int64_t k = static_cast<int64_t>(g) * 128 + lane * 4;
    const uint4 w = *reinterpret_cast<const uint4*>(packed + static_cast<int64_t>(r) * K + k);
    uint32_t affine = 0;                                   // of channel `lane`: the scale's byte, the byte of -z * s above it
    if (lane < 8) {
      const int64_t at = (static_cast<int64_t>(r) * 8 + lane) * kg + g;
      const int s = s4[at], z = z4[at];
      affine = (static_cast<uint32_t>(s) & 0xFFu) | ((static_cast<uint32_t>(-z * s) & 0xFFu) << 16);
    }
    // byte j of the four words (channels 2 j and 2 j + 1 at four k) gathered in one register
    const uint32_t ab = __byte_perm(w.x, w.y, 0x5140), cd = __byte_perm(w.z, w.w, 0x5140);
    const uint32_t ef = __byte_perm(w.x, w.y, 0x7362), gh = __byte_perm(w.z, w.w, 0x7362);
    const uint32_t tb[4] = {__byte_perm(ab, cd, 0x5410), __byte_perm(ab, cd, 0x7632),
                            __byte_perm(ef, gh, 0x5410), __byte_perm(ef, gh, 0x7632)};
    int8_t* dst = out + static_cast<int64_t>(r) * 8 * K + k;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint32_t a = __shfl_sync(0xffffffffu, affine, c), s = a & 0xFFu, z2 = __byte_perm(a, a, 0x3232);
      const uint32_t nib = tb[c >> 1] >> (4 * (c & 1));
      const uint32_t even = (nib & 0x000F000Fu) * s + z2, odd = ((nib >> 8) & 0x000F000Fu) * s + z2;
      *reinterpret_cast<uint32_t*>(dst + c * K) = __byte_perm(even, odd, 0x6240);
    }
  }
}

static int launch_w4a8_expand(const void* packed, const int8_t* s4, const int8_t* z4, void* out, int64_t rows8, int64_t K,
                              const ScaleCasts& casts, cudaStream_t st) {
  const int64_t groups = rows8 * (K / 128);
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((groups + 7) / 8, 148 * 32));
  auto go = [&](auto kernel) {
    kernel<<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(packed), s4, z4, static_cast<int8_t*>(out), rows8, K, casts);
  };
  // 32-bit indices where they suffice: the division per group is then a few instructions
  if (groups < (int64_t(1) << 31)) go(w4a8_expand_kernel<uint32_t>);
  else go(w4a8_expand_kernel<int64_t>);
  return check_launch("w4a8_expand_int8");
}

// Clears *ok where (q - z4) * s4 leaves int8 for a nibble that the weight holds.  One thread: 8 channels of one packed row and
// one 128-k group.  The packed words are only read where nibbles 0 and 15, the ends of the range, do not both stay inside
// (the product is linear in q): for weights from the quantizer the pass reads s4 and z4 alone.
__global__ void __launch_bounds__(256) w4a8_range_kernel(const uint32_t* __restrict__ packed, const int8_t* __restrict__ s4,
                                                         const int8_t* __restrict__ z4, int64_t rows8, int64_t K,
                                                         int32_t* __restrict__ ok) {
  const int64_t kg = K / 128, total = rows8 * kg;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / kg, g = i - r * kg;
    auto inside = [](int v) { return v >= -128 && v <= 127; };
    for (int c = 0; c < 8; ++c) {
      const int s = s4[(r * 8 + c) * kg + g], z = z4[(r * 8 + c) * kg + g];
      if (inside(-z * s) && inside((15 - z) * s)) continue;
      bool good = true;
      for (int j = 0; j < 128; ++j) good &= inside((static_cast<int>((packed[r * K + g * 128 + j] >> (4 * c)) & 0xF) - z) * s);
      if (!good) *ok = 0;
    }
  }
}

// One packed word = 8 consecutive k of one row -> 8 bf16.  A scale group is 16 words and rows are whole groups, so word i has
// scale i / 16 and its values stand at 8 i: no row or column is computed.  A thread takes kExpandWords words, 256 apart, whose
// loads are in flight together; a nibble becomes a float by an or with the bits of 2^23 instead of a conversion, which runs at
// a quarter of the rate.  8 experts of a Mixtral layer (gate/up 0.5 GB in, 1.9 GB out, then down): 689 + 348 us with a division per
// word and one word at a time, 514 + 261 us here.
constexpr int kExpandWords = 4;
__global__ void __launch_bounds__(256) w4a16_expand_kernel(const uint32_t* __restrict__ packed,
                                                           const __nv_bfloat16* __restrict__ scale,
                                                           const __nv_bfloat16* __restrict__ zero,
                                                           __nv_bfloat16* __restrict__ out, int64_t total) {
  constexpr float kTwo23 = 8388608.f;
  for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * (256 * kExpandWords) + threadIdx.x; i0 < total;
       i0 += static_cast<int64_t>(gridDim.x) * (256 * kExpandWords)) {
    uint32_t word[kExpandWords];
    float sc[kExpandWords], zp[kExpandWords];
#pragma unroll
    for (int u = 0; u < kExpandWords; ++u) {
      const int64_t i = i0 + u * 256;
      if (i >= total) break;
      word[u] = packed[i];
      sc[u] = __bfloat162float(scale[i >> 4]);
      zp[u] = __bfloat162float(zero[i >> 4]);
    }
#pragma unroll
    for (int u = 0; u < kExpandWords; ++u) {
      const int64_t i = i0 + u * 256;
      if (i >= total) break;
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = ((__uint_as_float(((word[u] >> (4 * j)) & 0xFu) | 0x4B000000u) - kTwo23) - zp[u]) * sc[u];
      store8(out + i * 8, v);
    }
  }
}

// Marlin-order symmetric int4 (fast_dequant/simple_marlin/utils.py:53-95): packed int32
// [K/16, N*16/8].  A packed row holds one 16-row k-tile, tiles of 16 x 16 flattened as
// n_tile*256 + k_in*16 + n_in, permuted in blocks of 1024 by `perm` (packed position i holds
// element perm[i]) and packed 8 nibbles per word.  Scales f16 [K/g, N] are permuted in blocks of
// 64 (grouped) or 32 (one group) columns; both permutations are closed forms (marlin_perm.cuh), so calls
// share no state.  One thread expands one word into
// out[n, k] = (q - 8) * s[k/g, n]  (f16, nn.Linear layout [N, K]).
__global__ void __launch_bounds__(256) marlin_expand_kernel(const uint32_t* __restrict__ packed,
                                                            const __half* __restrict__ s,
                                                            __half* __restrict__ out, int64_t K,
                                                            int64_t N, int64_t groupsize, int L) {
  const int64_t words_per_row = N * 2;
  const int64_t total = (K / 16) * words_per_row;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / words_per_row, j = i - r * words_per_row;
    const uint32_t word = packed[i];
#pragma unroll
    for (int f = 0; f < 8; ++f) {
      const int64_t pcol = j * 8 + f;
      const int64_t c = (pcol / 1024) * 1024 + marlin_perm(static_cast<int>(pcol % 1024));
      const int64_t n = (c / 256) * 16 + (c % 16);
      const int64_t k = r * 16 + (c % 256) / 16;
      const int64_t g = groupsize > 0 ? k / groupsize : 0;
      const float sc = __half2float(s[g * N + (n / L) * L + (L == 64 ? marlin_scale_inv64(static_cast<int>(n % L)) : marlin_scale_inv32(static_cast<int>(n % L)))]);
      const int q = static_cast<int>((word >> (4 * f)) & 0xF);
      out[n * K + k] = __float2half_rn(static_cast<float>(q - 8) * sc);
    }
  }
}

}  // namespace b200moe

using namespace b200moe;

extern "C" int b200moe_marlin_expand_f16(const void* packed, const void* scales_f16, void* out_f16,
                                         int64_t K, int64_t N, int64_t groupsize, void* stream) {
  B200MOE_REQUIRE(packed && scales_f16 && out_f16, B200MOE_BAD_ARG, "marlin_expand_f16: null pointer");
  B200MOE_REQUIRE(K > 0 && N > 0 && K % 16 == 0 && N % 64 == 0 && (N * 16) % 1024 == 0, B200MOE_BAD_SHAPE,
                  "marlin_expand_f16: Matrix dimensions not compatible with Marlin kernel requirements (K=%lld N=%lld)",
                  (long long)K, (long long)N);
  B200MOE_REQUIRE(groupsize == -1 || (groupsize > 0 && K % groupsize == 0), B200MOE_BAD_SHAPE,
                  "marlin_expand_f16: K dimension not divisible by groupsize: K=%lld, groupsize=%lld", (long long)K, (long long)groupsize);
  cudaStream_t st = as_stream(stream);
  const int scale_perm_len = groupsize == -1 ? 32 : 64;
  const int64_t total = (K / 16) * N * 2;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((total + 255) / 256, 148 * 32));
  marlin_expand_kernel<<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(packed), static_cast<const __half*>(scales_f16),
                                             static_cast<__half*>(out_f16), K, N, groupsize, scale_perm_len);
  return check_launch("marlin_expand_f16");
}

extern "C" int b200moe_w4a8_expand_int8(const void* packed, const int8_t* s4, const int8_t* z4, void* out,
                                        int64_t W, int64_t N, int64_t K, void* stream) {
  B200MOE_REQUIRE(packed && s4 && z4 && out, B200MOE_BAD_ARG, "w4a8_expand_int8: null pointer");
  B200MOE_REQUIRE(W >= 0 && N > 0 && K > 0 && N % 8 == 0 && K % 128 == 0, B200MOE_BAD_SHAPE,
                  "w4a8_expand_int8: N=%lld must be a multiple of 8 and K=%lld of 128", (long long)N, (long long)K);
  B200MOE_REQUIRE(aligned(packed, 16) && aligned(out, 4), B200MOE_BAD_ALIGN, "w4a8_expand_int8: alignment");
  if (W == 0) return B200MOE_OK;
  return launch_w4a8_expand(packed, s4, z4, out, W * (N / 8), K, ScaleCasts{}, as_stream(stream));
}

extern "C" int b200moe_w4a8_gemm_operands(const void* packed, const int8_t* s4, const int8_t* z4, void* out, int64_t N, int64_t K,
                                          const void* a_s_f16, float* a_s, int64_t a_s_count, const void* b_s_f16, float* b_s,
                                          int64_t b_s_count, void* stream) {
  B200MOE_REQUIRE(packed && s4 && z4 && out, B200MOE_BAD_ARG, "w4a8_gemm_operands: null pointer");
  B200MOE_REQUIRE(N > 0 && K > 0 && N % 8 == 0 && K % 128 == 0 && a_s_count >= 0 && b_s_count >= 0, B200MOE_BAD_SHAPE,
                  "w4a8_gemm_operands: N=%lld must be a multiple of 8 and K=%lld of 128", (long long)N, (long long)K);
  B200MOE_REQUIRE((a_s_count == 0 || (a_s_f16 && a_s)) && (b_s_count == 0 || (b_s_f16 && b_s)), B200MOE_BAD_ARG,
                  "w4a8_gemm_operands: null scales");
  B200MOE_REQUIRE(aligned(packed, 16) && aligned(out, 4) && aligned(a_s_f16, 2) && aligned(b_s_f16, 2) && aligned(a_s, 4) && aligned(b_s, 4),
                  B200MOE_BAD_ALIGN, "w4a8_gemm_operands: alignment");
  const ScaleCasts casts{{static_cast<const __half*>(a_s_f16), static_cast<const __half*>(b_s_f16)}, {a_s, b_s}, {a_s_count, b_s_count}};
  return launch_w4a8_expand(packed, s4, z4, out, N / 8, K, casts, as_stream(stream));
}

extern "C" int b200moe_w4a8_range_check(const void* packed, const int8_t* s4, const int8_t* z4, int64_t W, int64_t N,
                                        int64_t K, int32_t* ok, void* stream) {
  B200MOE_REQUIRE(packed && s4 && z4 && ok, B200MOE_BAD_ARG, "w4a8_range_check: null pointer");
  B200MOE_REQUIRE(W >= 0 && N > 0 && K > 0 && N % 8 == 0 && K % 128 == 0, B200MOE_BAD_SHAPE,
                  "w4a8_range_check: N=%lld must be a multiple of 8 and K=%lld of 128", (long long)N, (long long)K);
  if (W == 0) return B200MOE_OK;
  const int64_t rows8 = W * (N / 8), total = rows8 * (K / 128);
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((total + 255) / 256, 148 * 32));
  w4a8_range_kernel<<<grid, 256, 0, as_stream(stream)>>>(static_cast<const uint32_t*>(packed), s4, z4, rows8, K, ok);
  return check_launch("w4a8_range_check");
}

extern "C" int b200moe_w4a16_expand_bf16(const void* packed, const void* scale_bf16, const void* zero_bf16,
                                         void* out_bf16, int64_t rows, int64_t K, void* stream) {
  B200MOE_REQUIRE(packed && scale_bf16 && zero_bf16 && out_bf16, B200MOE_BAD_ARG, "w4a16_expand_bf16: null pointer");
  B200MOE_REQUIRE(rows >= 0 && K > 0 && K % 128 == 0, B200MOE_BAD_SHAPE, "w4a16_expand_bf16: K=%lld must be a multiple of 128", (long long)K);
  B200MOE_REQUIRE(aligned(out_bf16, 16), B200MOE_BAD_ALIGN, "w4a16_expand_bf16: alignment");
  if (rows == 0) return B200MOE_OK;
  const int64_t total = rows * (K / 8);
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((total + 256 * kExpandWords - 1) / (256 * kExpandWords), 148 * 32));
  w4a16_expand_kernel<<<grid, 256, 0, as_stream(stream)>>>(static_cast<const uint32_t*>(packed),
                                                           static_cast<const __nv_bfloat16*>(scale_bf16),
                                                           static_cast<const __nv_bfloat16*>(zero_bf16),
                                                           static_cast<__nv_bfloat16*>(out_bf16), total);
  return check_launch("w4a16_expand_bf16");
}
