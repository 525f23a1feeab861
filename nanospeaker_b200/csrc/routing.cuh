// Pieces shared by the routing kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace moe {

constexpr int MAX_EXPERTS = 256;  // router + dispatch kernels keep per-expert state on chip
constexpr int MAX_TOPK = 16;
constexpr int ALIGN_M = 128;     // expert runs are padded to whole 128-row GEMM tiles

// Order-preserving map fp32 -> uint32 (larger float -> larger key); NaN sorts above +inf and
// -0.0 ties with +0.0, so ties between equal values fall to the lowest expert index below.
__device__ __forceinline__ uint32_t float_key(float f) {
  if (f != f) return 0xFFFFFFFFu;
  if (f == 0.f) f = 0.f;
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

}  // namespace moe

#include <cuda_bf16.h>

namespace moe {
// router_fused.cu: router top-k in chunked mode (block b owns tokens [b * tokens_per_block, ...))
// that also leaves the dispatch's per-block histograms and the sentinel fill. Returns an error code
// of include/moe_b200.h.
// With `sc` given and few enough blocks for one cluster, the four-lanes-per-token kernel also runs the
// dispatch's second pass itself and *did_scatter is set: no further launch is needed.
// What a forward reports besides its output, made where the counts are: the routed experts' counts for
// the caller, the balance loss coef * E * sum_e (counts[e] / sum counts) * (colsum[e] / T) -- the
// arithmetic of moe_b200_balance_loss, same order -- or zero when it is off (colsum null), and with a
// capacity the number of pairs over it.
struct FinishArgs {
  int32_t* counts;        // null: nothing of this
  const float* colsum;
  float* aux;
  int64_t* dropped;       // may be null
  int64_t n_tokens;
  float coef;
  int32_t n_experts, aux_is_16bit;
  // The 128-row tiles in an order that keeps together what belongs to neighbouring tokens: a run's rows are
  // in token order, so its tiles are cut into `windows` (a power of two) equal parts, and window by window
  // come every routed expert's; the shared experts' tiles follow. (tile, owner); null: not made.
  int2* order;
  int32_t windows;
};
struct ScatterArgs {
  int32_t* counts;
  int32_t* pad_offsets;
  int32_t* n_post_pad;
  int32_t* expert_ids;
  int64_t n_tiles_cap;
  int32_t* inv_ids;
  int32_t capacity;   // > 0: experts below n_capped keep the first `capacity` pairs of their runs
  int32_t n_capped;
  FinishArgs fin;
};
int launch_router_fused_chunked(const __nv_bfloat16* logits, int ld, const float* bias,
                                const float* noise,
                                int64_t n_tokens, int n_experts, int top_k, int n_shared,
                                int normalize, int full_softmax, __nv_bfloat16* w_all,
                                int64_t* idx_all, float* colsum, int tokens_per_block, int n_blocks,
                                int32_t* block_hist, int32_t* sorted_ids, int64_t l_cap,
                                cudaStream_t st, const ScatterArgs* sc = nullptr,
                                bool* did_scatter = nullptr);
// routing.cu: moe_b200_router_dispatch with an expert capacity (0 = dropless) on the first n_experts
// experts and the forward's reports; *launches (may be null) receives the number of kernels.
int router_dispatch(const void* logits, int32_t ld, const float* bias, const float* noise,
                    int64_t n_tokens, int32_t n_experts, int32_t top_k, int32_t n_shared,
                    int32_t normalize, int32_t full_softmax, void* w_all, int64_t* idx_all,
                    float* colsum, int32_t* sorted_ids, int32_t* expert_ids, int32_t* pad_offsets,
                    int32_t* counts, int32_t* n_post_pad, int32_t* inv_ids, void* scratch,
                    size_t scratch_bytes, int32_t capacity, const FinishArgs& fin, int32_t* status,
                    void* stream, int* launches);
// router_front.cu: everything up to the plan for a small batch, from the token rows and the router weight
// [D, E] as it is. Two launches; results as of the logits GEMM and router_dispatch.
struct FrontCall {
  const void *x, *router_w;
  const float *bias, *noise;
  int64_t n_tokens;
  int32_t d_model, n_experts, n_shared, top_k, normalize, full_softmax;
  void* w_all;
  int64_t* idx_all;
  void *logits, *w_padded;   // [T, ld], [D, ld] with zeros past E: for a backward; null: not written
  int32_t ld;
  int32_t* sorted_ids;
  ScatterArgs scatter;       // its n_tiles_cap tells l_cap
  void* scratch;
  int32_t* status;
};
bool router_front_covers(int64_t n_tokens, int32_t d_model, int32_t n_experts, int32_t n_shared,
                         int32_t top_k, const void* x, const void* router_w);
size_t router_front_scratch_bytes(int64_t n_tokens, int32_t n_experts, int32_t n_shared);
int router_front(const FrontCall& c, cudaStream_t st);
// router_fused.cu: moe_b200_router_fused_bwd with two more inputs. extra_dw [T, extra_ld] bf16: what
// d(topk_w) of a pair gains, read at its expert's column; inv_ids [T * (k + S)]: pairs without a slot
// (dropped by a capacity) have no d(topk_w). Either may be null.
int router_fused_bwd(const void* logits, int32_t ld, const float* bias, const float* noise,
                     const int64_t* idx_all, const void* dw_all, const void* extra_dw,
                     int32_t extra_ld, const int32_t* inv_ids, int64_t n_tokens, int32_t n_experts,
                     int32_t top_k, int32_t n_shared, int32_t normalize, int32_t full_softmax,
                     const float* d_aux, const int32_t* counts, float aux_coef, void* d_logits,
                     int32_t ld_out, void* stream);
}  // namespace moe
