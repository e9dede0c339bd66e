// Shared host/device helpers for the b200moe library.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "../../include/b200moe.h"

namespace b200moe {

// Records a message for b200moe_last_error() and returns `status`.
int fail(int status, const char* fmt, ...);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Returns B200MOE_OK or records the CUDA launch error.
int check_launch(const char* what);

// The error of a refused call, taken from the runtime too: what it keeps would be reported by the next launch.
inline int refused(const char* what, cudaError_t e) {
  cudaGetLastError();
  return fail(B200MOE_LAUNCH_FAILED, "%s: %s", what, cudaGetErrorString(e));
}

// Opts a kernel in to `bytes` of dynamic shared memory on the current device, once per kernel and device.
int set_dynamic_smem(const void* kernel, size_t bytes);

// b200moe_grouped_gemm_bf16 (gemm_fp8.cu) on one group of all M rows, which needs no group table; a [M, K] contiguous.
int dense_gemm_bf16(const void* a, const void* b, void* c, int64_t c_row_stride_bytes, int64_t M, int64_t N, int64_t K,
                    int epilogue, int32_t* status_word, void* stream);

// Programmatic dependent launch.  launch_dependent() lets the kernel's blocks start while the kernel before it in the stream
// drains; wait_for_predecessors() then holds them until that kernel is complete and its writes are visible.  A kernel that is
// launched this way must call it before it touches global memory, reads and writes alike (its output may be what the kernel
// before it still reads); since every one of them does, completion is transitive along the stream.
// allow_dependents() says that this block needs no more of the machine than it has: once all blocks have said so or left, the
// next kernel's blocks may take what is free.  The GEMM kernels do not say so: their CTAs leave no room beside them, and with
// the next kernel let in early they were slower (fp8 linear layer of 16 rows 18.0 -> 19.7 us, small fp8 layer of 512 tokens 69.9
// -> 72.2).
__device__ __forceinline__ void wait_for_predecessors() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
int launch_dependent(const char* what, void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return e == cudaSuccess ? check_launch(what) : refused(what, e);
}

// Router logits of few tokens on the CUDA cores (router.cu), from the operands of b200moe_router_logits_bf16x3 (gemm_fp8.cu).
// us without the selection, weight out of memory, tensor cores with 16 splits -> here: hidden size 7168, 256 experts 18.6 -> 14.4 for
// one token, 18.5 -> 14.3 for two, 18.8 -> 22.5 for four; 4096 and 128 rows 14.3 -> 10.3, 14.3 -> 10.2, 14.4 -> 16.4; 1024 and 128 rows
// 11.1 -> 6.3 for one, 10.4 -> 8.2 for two.
constexpr int64_t kRouterFewTokens = 2;
int router_logits_few(const void* x_bf16, const void* w3_bf16, float* logits, int64_t T, int64_t H, int E, cudaStream_t st);

#define B200MOE_REQUIRE(cond, status, ...)                 \
  do {                                                     \
    if (!(cond)) return ::b200moe::fail((status), __VA_ARGS__); \
  } while (0)

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// ---- device-side element access ------------------------------------------------
template <typename T> struct Vec8;  // eight elements of T as one vector load

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __half* p, float (&v)[8]) {
  const uint4 r = *reinterpret_cast<const uint4*>(p);
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    v[2 * i] = f.x; v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 r = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x; v[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store8(__half* p, const float (&v)[8]) {
  uint4 r;
  __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = r;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&v)[8]) {
  uint4 r;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = r;
}

// Round-to-nearest-even e4m3 with saturation to +-448; NaN stays NaN (0x7f).
__device__ __forceinline__ uint8_t to_e4m3(float v) {
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}
// Packs eight floats as eight e4m3 bytes (element 0 in the lowest byte).
__device__ __forceinline__ uint2 pack8_e4m3(const float (&v)[8]) {
  uint2 r;
  const uint32_t a = __nv_cvt_float2_to_fp8x2(make_float2(v[0], v[1]), __NV_SATFINITE, __NV_E4M3);
  const uint32_t b = __nv_cvt_float2_to_fp8x2(make_float2(v[2], v[3]), __NV_SATFINITE, __NV_E4M3);
  const uint32_t c = __nv_cvt_float2_to_fp8x2(make_float2(v[4], v[5]), __NV_SATFINITE, __NV_E4M3);
  const uint32_t d = __nv_cvt_float2_to_fp8x2(make_float2(v[6], v[7]), __NV_SATFINITE, __NV_E4M3);
  r.x = a | (b << 16);
  r.y = c | (d << 16);
  return r;
}
__device__ __forceinline__ float e4m3_to_float(uint8_t b) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(b, __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}

__device__ __forceinline__ float round_to(float v, __nv_bfloat16) {
  return __bfloat162float(__float2bfloat16_rn(v));
}
__device__ __forceinline__ float round_to(float v, __half) {
  return __half2float(__float2half_rn(v));
}
__device__ __forceinline__ float round_to(float v, float) { return v; }

}  // namespace b200moe
