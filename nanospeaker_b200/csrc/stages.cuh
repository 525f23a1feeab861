// Stages of the block with options that the C entry points of the same names do not have (gemm.cu).
#pragma once
#include <stdint.h>
#include <vector_types.h>

namespace moe {
// moe_b200_up_gemm / moe_b200_dhidden_glu_bwd with gathered rows (gather_top_k > 0) that are also written
// in slot order to rows_out [rows, d_model] (null: not), the routed experts' runs only: what
// moe_b200_permute up to the first shared run would have written.
int up_gemm(const void* a, int64_t rows, int32_t d_model, const void* w_in, int32_t n_groups,
            const void* w_extra, int32_t n_extra, int32_t d_hidden, const int32_t* expert_ids,
            const int32_t* n_post_pad, int32_t n_fixed_groups, const int32_t* sorted_ids,
            int32_t gather_top_k, int64_t n_pairs, int32_t activation, void* hid, void* raw,
            const void* a_tokens, int64_t n_tokens, const int32_t* pad_offsets, const void* bias,
            void* rows_out, const int2* order, int32_t* status, void* stream);
// (order: FinishArgs::order, or null; moe_b200_down_gemm_acc with it:)
int down_gemm_acc(const void* hid, int64_t rows, int32_t k_dim, const void* w_out, int32_t n_groups,
                  const void* w_extra, int32_t n_extra, int32_t d_model, const int32_t* expert_ids,
                  const int32_t* n_post_pad, int32_t n_fixed_groups, const int32_t* sorted_ids,
                  const void* pair_w, int64_t n_pairs, int32_t top_k, void* acc, int64_t n_tokens,
                  const void* bias, const int2* order, int32_t* status, void* stream);
int dhidden_glu_bwd(const void* douts, int64_t rows, int32_t d_model, const void* w_out,
                    int32_t n_groups, const void* w_extra, int32_t n_extra,
                    int32_t d_hidden, const int32_t* expert_ids,
                    const int32_t* n_post_pad, int32_t n_fixed_groups,
                    const int32_t* sorted_ids, int32_t gather_top_k, const void* pair_w,
                    int64_t n_pairs, const void* a1, int32_t activation, void* da1,
                    void* hidw, void* dtw, const void* dout_tokens, int64_t n_tokens,
                    const int32_t* pad_offsets, void* rows_out, int32_t* status, void* stream);
// moe_b200_down_gemm_sum with addend [n_tokens, d_model] (may be null) added to the sum.
int down_gemm_sum(const void* hid, int64_t rows, int32_t k_dim, const void* w_out,
                  int32_t n_sum, int32_t d_model, const int32_t* run_offsets,
                  int64_t n_tokens, const void* addend, void* out, int32_t* status, void* stream);
// moe_b200_dx_gemm_acc, on the routed schedule with pad_offsets also adding the router's share, dl
// [n_tokens, ld] @ router_w^T (router_w [d_model, ld], ld a multiple of 64; dl may be null).
int dx_gemm_acc(const void* da1, int64_t rows, int32_t d_hidden, const void* w_in,
                int32_t n_groups, const void* w_extra, int32_t n_extra, int32_t d_model,
                const int32_t* expert_ids, const int32_t* n_post_pad, int32_t n_fixed_groups,
                const int32_t* sorted_ids, int64_t n_pairs, int32_t top_k, void* acc, int64_t n_tokens,
                const int32_t* pad_offsets, const void* dl, const void* router_w, int32_t ld,
                int32_t* status, void* stream);
// moe_b200_wgrad with what the caller knows beside: no run is longer than max_run rows, and dw has
// out_cols columns (other than n_dim: one fixed group of more than the rows of a chunk).
int wgrad(const void* a, int32_t a_grouped, int32_t m_dim, const void* b,
          int32_t b_grouped, int32_t n_dim, int64_t rows, const int32_t* pad_offsets,
          int32_t n_groups, int32_t ks_rows, const int32_t* sorted_ids,
          int32_t gather_top_k, int64_t n_pairs, int32_t gather_which, void* dw,
          int32_t n_first, void* dw_extra, void* partials, size_t partial_bytes,
          const void* alt, int64_t alt_rows, int32_t alt_which, int64_t max_run, int32_t out_cols, int32_t* status,
          void* stream);
// Rows per split-K chunk for runs of at most max_run rows. moe_b200_wgrad picks it with max_run = rows.
int wgrad_chunk_rows(int32_t m_dim, int32_t n_dim, int64_t rows, int32_t n_groups, int32_t routed,
                     int64_t max_run);
}  // namespace moe
