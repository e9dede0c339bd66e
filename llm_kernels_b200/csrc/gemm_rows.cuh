// The GEMMs for few rows per group (gemm_fp8_rows.cu): interface for the dispatch in gemm_fp8.cu.
#pragma once

#include "common.cuh"

namespace b200moe {
namespace rows {

constexpr int kRowsChunk = 64;         // tokens per tile at most
// Average rows per group up to which gemm_fp8.cu hands over.  64 experts, gate/up + down of a DeepSeek-V3 layer, us (128-token
// tiles -> these): 4 rows 522 -> 441, 16 rows 535 -> 468, 32 rows 549 -> 532, 48 rows 555 -> 595; with Zipf-skewed rows
// 16 on average 558 -> 535, 32 on average 580 -> 640.  Other shapes at 24 rows: 8 experts of N 28672 K 4096 248 -> 203, of
// N 4096 K 14336 112 -> 112; 256 of N 1024 K 1024 134 -> 103; one weight of N 4096 K 7168 50 -> 41.
constexpr int kMaxRowsPerGroup = 24;

int launch_fp8(const void* a, int64_t a_stride, const float* a_s, int64_t a_s_stride, const void* b, const float* b_s, void* c,
               int c_dtype, int64_t c_stride, float* c_s, int64_t c_s_stride, int64_t M_total, int64_t N, int64_t K, int num_groups,
               int num_weights, const int64_t* seg, const int64_t* widx, int fused, int act, int32_t* status, cudaStream_t st);

}  // namespace rows
}  // namespace b200moe
