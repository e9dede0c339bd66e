// One forward pass of a single-rank MoE layer (moe/all2all_moe.py:167-184: gate, experts, shared experts) as one host
// call: the launches below follow each other on the caller's stream and nothing is read back.
//
// Issued from Python one by one, the same launches cost about 20 us of interpreter time each (argument conversion,
// views, allocator calls): 210 us per pass, more than the kernels of a decode step need.
#include <algorithm>

#include "common.cuh"

namespace b200moe {

// Workspace of a pass of T tokens: offsets in bytes, each 256-byte aligned.
struct LayerPlan {
  int64_t S, rec, rec_scale;        // slots, bytes of a permuted row, byte offset of its scales
  int ksplits;
  int64_t idx, wts, ids, dst, seg, scratch, scratch_bytes, part, send, h, h_s, down, shared_h, total;
};

static LayerPlan plan_layer(const b200moe_layer& L, int64_t T) {
  LayerPlan p{};
  const int64_t H = L.hidden, I = L.inter;
  p.S = T * L.top_k;
  p.rec_scale = H;
  p.rec = L.method == B200MOE_LAYER_W4A16 ? 2 * H : (H + H / 128 * 4 + 15) / 16 * 16;
  p.ksplits = b200moe_router_ksplits(T, H, L.router_rows);
  int64_t off = 0;
  auto take = [&](int64_t bytes) { const int64_t o = off; off += (std::max<int64_t>(bytes, 16) + 255) / 256 * 256; return o; };
  p.idx = take(p.S * 8);
  p.wts = take(p.S * 4);
  p.ids = take(p.S * 8);
  p.dst = take(p.S * 4);
  p.seg = take((L.experts + 1) * 8);
  p.scratch_bytes = static_cast<int64_t>(b200moe_route_metadata_workspace_bytes(p.S, L.experts));
  p.scratch = take(p.scratch_bytes);
  p.part = take(p.ksplits * T * L.router_rows * 4);
  p.send = take(p.S * p.rec);
  p.h = take(p.S * I * (L.method == B200MOE_LAYER_W4A16 ? 2 : 1));
  p.h_s = take(p.S * (I / 128) * 4);
  p.down = take(p.S * H * 2);
  p.shared_h = take(L.shared_inter ? T * L.shared_inter * 2 : 0);
  p.total = off;
  return p;
}

static int check_layer(const b200moe_layer* L) {
  B200MOE_REQUIRE(L && L->struct_bytes == sizeof(b200moe_layer), B200MOE_BAD_ARG, "layer: descriptor size");
  B200MOE_REQUIRE(L->method >= B200MOE_LAYER_FP8 && L->method <= B200MOE_LAYER_W4A8, B200MOE_BAD_ARG, "layer: method %d", L->method);
  B200MOE_REQUIRE(L->hidden > 0 && L->hidden % 128 == 0 && L->inter > 0 && L->inter % 128 == 0, B200MOE_BAD_SHAPE,
                  "layer: hidden and intermediate sizes must be multiples of 128");
  B200MOE_REQUIRE(L->experts >= 1 && L->top_k >= 1 && L->top_k <= L->experts && L->router_rows >= L->experts &&
                  L->shared_inter >= 0, B200MOE_BAD_SHAPE, "layer: %d experts, top-%d", L->experts, L->top_k);
  return B200MOE_OK;
}

}  // namespace b200moe

using namespace b200moe;

extern "C" int64_t b200moe_layer_workspace_bytes(const b200moe_layer* L, int64_t T) {
  if (check_layer(L) || T < 0) return -1;
  return plan_layer(*L, T).total;
}

extern "C" int b200moe_layer_workspace_layout(const b200moe_layer* L, int64_t T, int64_t* send, int64_t* seg) {
  if (int rc = check_layer(L)) return rc;
  const LayerPlan p = plan_layer(*L, T);
  *send = p.send;
  *seg = p.seg;
  return B200MOE_OK;
}

// A side stream's part in one pass: forked from the pass's stream and joined to it on every way out, with events of its own,
// since other passes may be using the same side stream.
class SideWork {
 public:
  explicit SideWork(cudaStream_t main) : main_(main) {}
  ~SideWork() {
    join();
    if (fork_) cudaEventDestroy(fork_);      // released by the runtime once the work recorded in them is through
    if (done_) cudaEventDestroy(done_);
  }
  int fork(cudaStream_t side) {
    side_ = side;
    if (int rc = check(cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming))) return rc;
    if (int rc = check(cudaEventCreateWithFlags(&done_, cudaEventDisableTiming))) return rc;
    if (int rc = check(cudaEventRecord(fork_, main_))) return rc;
    if (int rc = check(cudaStreamWaitEvent(side_, fork_, 0))) return rc;
    forked_ = true;
    return B200MOE_OK;
  }
  int done() {                               // what the side stream holds now is what the pass waits for
    recorded_ = true;
    return check(cudaEventRecord(done_, side_));
  }
  int join() {
    if (!forked_) return B200MOE_OK;
    forked_ = false;
    if (!recorded_) if (int rc = done()) return rc;
    return check(cudaStreamWaitEvent(main_, done_, 0));
  }

 private:
  static int check(cudaError_t e) {
    return e == cudaSuccess ? B200MOE_OK : fail(B200MOE_LAUNCH_FAILED, "layer_forward: side stream: %s", cudaGetErrorString(e));
  }
  cudaStream_t main_, side_ = nullptr;
  cudaEvent_t fork_ = nullptr, done_ = nullptr;
  bool forked_ = false, recorded_ = false;
};

#define STEP(call) do { if (int rc_ = (call)) return rc_; } while (0)

extern "C" int b200moe_layer_forward(const b200moe_layer* Lp, const void* x, void* y, int64_t T, void* workspace,
                                     int64_t workspace_bytes, void* stream) {
  if (int rc = check_layer(Lp)) return rc;
  const b200moe_layer& L = *Lp;
  B200MOE_REQUIRE(T >= 0 && T * L.top_k < (int64_t(1) << 31), B200MOE_BAD_SHAPE, "layer_forward: T=%lld", (long long)T);
  if (T == 0) return B200MOE_OK;
  B200MOE_REQUIRE(x && y && workspace && aligned(workspace, 256), B200MOE_BAD_ARG, "layer_forward: null pointer or workspace alignment");
  const LayerPlan p = plan_layer(L, T);
  B200MOE_REQUIRE(workspace_bytes >= p.total, B200MOE_WORKSPACE_TOO_SMALL, "layer_forward: workspace %lld < %lld bytes",
                  (long long)workspace_bytes, (long long)p.total);
  char* ws = static_cast<char*>(workspace);
  const int64_t H = L.hidden, I = L.inter;
  auto* idx = reinterpret_cast<int64_t*>(ws + p.idx);
  auto* wts = reinterpret_cast<float*>(ws + p.wts);
  auto* dst = reinterpret_cast<int32_t*>(ws + p.dst);
  auto* seg = reinterpret_cast<int64_t*>(ws + p.seg);
  auto* part = reinterpret_cast<float*>(ws + p.part);
  char* send = ws + p.send;
  auto* send_s = reinterpret_cast<float*>(send + p.rec_scale);
  void* h = ws + p.h;
  auto* h_s = reinterpret_cast<float*>(ws + p.h_s);
  void* down = ws + p.down;
  SideWork side(as_stream(stream));

  STEP(b200moe_router_logits_bf16x3(x, L.router_w3, part, T, H, L.router_rows, p.ksplits, stream));
  STEP(b200moe_router_select(part, p.ksplits, L.router_rows, L.router_bias, T, L.experts, L.top_k, L.n_group, L.topk_group,
                             L.scoring, L.norm_topk_prob, L.scaling, idx, wts, stream));
  if (L.shared_inter) {
    // gate/up of the shared experts needs only x: on the side stream it fills the SMs the routed path leaves idle
    STEP(side.fork(as_stream(L.side_stream)));
    STEP(dense_gemm_bf16(x, L.shared_w13, ws + p.shared_h, 2 * L.shared_inter, T, 2 * L.shared_inter, H, L.act ? 5 : 2, L.status,
                         L.side_stream));
    STEP(side.done());
  }
  STEP(b200moe_route_metadata(idx, p.S, L.experts, reinterpret_cast<int64_t*>(ws + p.ids), dst, seg, ws + p.scratch,
                              static_cast<size_t>(p.scratch_bytes), stream));
  const int E = L.experts;
  switch (L.method) {
    case B200MOE_LAYER_FP8:
      STEP(b200moe_permute_quant_fp8(x, B200MOE_BF16, dst, idx, 0, E - 1, T, L.top_k, H, send, p.rec, send_s, p.rec / 4, stream));
      STEP(b200moe_grouped_gemm_fp8(send, p.rec, send_s, p.rec / 4, L.w13, static_cast<const float*>(L.w13_scale), h,
                                    B200MOE_FP8_E4M3, I, h_s, I / 128, p.S, 2 * I, H, E, E, seg, nullptr, L.act ? 4 : 1,
                                    nullptr, nullptr, L.status, nullptr, stream));
      STEP(b200moe_grouped_gemm_fp8(h, I, h_s, I / 128, L.w2, static_cast<const float*>(L.w2_scale), down, B200MOE_BF16, 2 * H,
                                    nullptr, 0, p.S, H, I, E, E, seg, nullptr, 0, nullptr, nullptr, L.status, nullptr, stream));
      break;
    case B200MOE_LAYER_W4A16:
      STEP(b200moe_pre_reorder(x, B200MOE_BF16, send, B200MOE_BF16, dst, idx, nullptr, 0, E - 1, T, L.top_k, H, stream));
      STEP(b200moe_grouped_gemm_w4a16(send, 2 * H, L.w13, L.w13_pairs, h, B200MOE_BF16, 2 * I, p.S, 2 * I, H, E, E, seg, nullptr,
                                      L.act ? 5 : 2, L.status, stream));
      STEP(b200moe_grouped_gemm_w4a16(h, 2 * I, L.w2, L.w2_pairs, down, B200MOE_BF16, 2 * H, p.S, H, I, E, E, seg, nullptr, 0,
                                      L.status, stream));
      break;
    default:
      STEP(b200moe_permute_quant_int8(x, B200MOE_BF16, dst, idx, 0, E - 1, T, L.top_k, H, send, p.rec, send_s, p.rec / 4, 1, stream));
      STEP(b200moe_grouped_gemm_w4a8(send, p.rec, send_s, p.rec / 4, L.w13, L.w13_pairs, static_cast<const float*>(L.w13_scale), h,
                                     B200MOE_I8, I, h_s, I / 128, p.S, 2 * I, H, E, E, seg, nullptr, L.act ? 4 : 1, L.status, stream));
      STEP(b200moe_grouped_gemm_w4a8(h, I, h_s, I / 128, L.w2, L.w2_pairs, static_cast<const float*>(L.w2_scale), down, B200MOE_BF16,
                                     2 * H, nullptr, 0, p.S, H, I, E, E, seg, nullptr, 0, L.status, stream));
      break;
  }
  STEP(b200moe_post_reorder(down, B200MOE_BF16, y, dst, idx, wts, 0, E - 1, T, L.top_k, H, stream));
  if (L.shared_inter) {
    STEP(side.join());
    STEP(dense_gemm_bf16(ws + p.shared_h, L.shared_w2, y, 2 * H, T, H, L.shared_inter, 3, L.status, stream));
  }
  return B200MOE_OK;
}
