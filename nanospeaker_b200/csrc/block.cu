// The whole block's forward and backward as ONE host call each: the stage sequence of
// nanospeaker_b200/moe_kernel.py (router GEMM, routing + dispatch, gather + up/gate GEMM + GLU,
// down GEMM, combine, balance loss; and the backward with its three independent
// branches on three streams) issued from C++, for hosts that pay per call into this library -- a
// Python caller's ~22 ctypes calls per step cost it more than the GPU needs for the work.
// Everything here is host code over the other entry points of include/moe_b200.h, plus a few
// trivial kernels: zero / copy a few words (memset and device-to-device copy nodes go to a copy
// engine, where they queue behind a caller's large host-to-device copy in flight: the end-to-end
// step lost 13 us to that), and the forward's first launch, which folds what would otherwise be small
// launches of their own on the critical path (pad the router weight, stack the biases, clear the
// column sums). All of them wait for their predecessors programmatically like the library's other
// kernels, so none of them breaks the chain of early launches.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/moe_b200.h"
#include "pdl.cuh"
#include "routing.cuh"
#include "stages.cuh"

namespace {

__global__ void zero_words_kernel(uint32_t* dst, int64_t n) {
  moe::pdl_trigger();
  moe::pdl_wait();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    dst[i] = 0u;
}
__global__ void copy_words_kernel(const uint32_t* src, uint32_t* dst, int64_t n) {
  moe::pdl_trigger();
  moe::pdl_wait();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    dst[i] = src[i];
}
inline int zero_words(void* dst, int64_t n_words, cudaStream_t st) {
  const int64_t blocks = (n_words + 255) / 256;
  moe::launch_pdl(zero_words_kernel, dim3(unsigned(blocks < 592 ? blocks : 592)), dim3(256), 0, st,
                  static_cast<uint32_t*>(dst), n_words);
  return cudaGetLastError() == cudaSuccess ? MOE_B200_OK : MOE_B200_ERR_CUDA;
}
inline int copy_words(const void* src, void* dst, int64_t n_words, cudaStream_t st) {
  const int64_t blocks = (n_words + 255) / 256;
  moe::launch_pdl(copy_words_kernel, dim3(unsigned(blocks < 592 ? blocks : 592)), dim3(256), 0, st,
                  static_cast<const uint32_t*>(src), static_cast<uint32_t*>(dst), n_words);
  return cudaGetLastError() == cudaSuccess ? MOE_B200_OK : MOE_B200_ERR_CUDA;
}

// The forward's first launch: up to PREP_JOBS small 16-bit matrices copied into zero-padded places
// (the router weight [D, E] -> [D, ld] as the tensor maps want it; the biases of both weight stacks
// one under the other) and, in the same launch, the column sums of the balance loss cleared.
constexpr int PREP_JOBS = 6;
struct PrepJob {
  const uint16_t* src;      // null: zeros
  uint16_t* dst;
  int32_t rows, cols;       // of src
  int32_t dst_rows, dst_ld; // of dst; what src does not cover is zero
};
struct PrepArgs {
  PrepJob job[PREP_JOBS];
  int32_t n_jobs;
  int32_t n_clear;
  float* clear;
};
__global__ void __launch_bounds__(256) prep_kernel(const PrepArgs a) {
  moe::pdl_trigger();
  moe::pdl_wait();
  const int first = int(blockIdx.x * blockDim.x + threadIdx.x);
  const int step = int(gridDim.x * blockDim.x);
  for (int i = first; i < a.n_clear; i += step) a.clear[i] = 0.f;
  for (int k = 0; k < a.n_jobs; ++k) {
    const PrepJob j = a.job[k];
    const int total = j.dst_rows * j.dst_ld;
    for (int i = first; i < total; i += step) {
      const int r = i / j.dst_ld, c = i - r * j.dst_ld;
      j.dst[i] = j.src != nullptr && r < j.rows && c < j.cols ? j.src[r * j.cols + c] : uint16_t(0);
    }
  }
}
inline int prep(const PrepArgs& a, cudaStream_t st) {
  int64_t most = a.n_clear;
  for (int k = 0; k < a.n_jobs; ++k)
    most = std::max(most, int64_t(a.job[k].dst_rows) * a.job[k].dst_ld);
  if (most > INT32_MAX) return MOE_B200_ERR_SHAPE;
  const int64_t blocks = std::min<int64_t>((most + 255) / 256, 148 * 8);
  moe::launch_pdl(prep_kernel, dim3(unsigned(std::max<int64_t>(blocks, 1))), dim3(256), 0, st, a);
  return cudaGetLastError() == cudaSuccess ? MOE_B200_OK : MOE_B200_ERR_CUDA;
}

// fp32 -> bf16 (the bias gradients' last step).
__global__ void __launch_bounds__(256)
    to_bf16_kernel(const float* src, __nv_bfloat16* dst, int32_t n) {
  moe::pdl_trigger();
  moe::pdl_wait();
  for (int i = int(blockIdx.x * blockDim.x + threadIdx.x); i < n; i += int(gridDim.x * blockDim.x))
    dst[i] = __float2bfloat16(src[i]);
}
inline int to_bf16(const float* src, void* dst, int32_t n, cudaStream_t st) {
  const int blocks = std::min((n + 255) / 256, 592);
  moe::launch_pdl(to_bf16_kernel, dim3(unsigned(blocks)), dim3(256), 0, st, src,
                  static_cast<__nv_bfloat16*>(dst), n);
  return cudaGetLastError() == cudaSuccess ? MOE_B200_OK : MOE_B200_ERR_CUDA;
}

constexpr size_t ALIGN = 256;
inline size_t up(size_t n) { return (n + ALIGN - 1) / ALIGN * ALIGN; }
inline int32_t router_ld(int32_t n_experts) { return (n_experts + 63) / 64 * 64; }

struct Carver {   // hands out aligned pieces of one caller-provided buffer
  char* base;
  size_t used = 0;
  explicit Carver(void* p) : base(static_cast<char*>(p)) {}
  void* take(size_t bytes) {
    void* r = base ? base + used : nullptr;
    used += up(bytes);
    return r;
  }
};

struct Sizes {
  int32_t ld, ks, n_all;
  int64_t m, l_cap;
};
inline Sizes sizes(int64_t n_tokens, int32_t n_experts, int32_t n_shared, int32_t top_k) {
  Sizes s;
  s.ld = router_ld(n_experts);
  s.ks = top_k + n_shared;
  s.n_all = n_experts + n_shared;
  s.m = n_tokens * s.ks;
  s.l_cap = moe_b200_l_cap(s.m, s.n_all);
  return s;
}

// A token has a row in a run once at most, and runs are padded to whole tiles.
inline int64_t longest_run(int64_t n_tokens) { return (n_tokens + 127) / 128 * 128; }
// Rows per split-K chunk of the three weight gradients.
struct Chunks {
  int32_t in, out, router;
};
inline Chunks chunks_of(const Sizes& z, int64_t n_tokens, int32_t d_model, int32_t d_hidden) {
  return Chunks{
      moe::wgrad_chunk_rows(d_model, 2 * d_hidden, z.l_cap, z.n_all, 1, longest_run(n_tokens)),
      moe::wgrad_chunk_rows(d_hidden, d_model, z.l_cap, z.n_all, 1, longest_run(n_tokens)),
      moe::wgrad_chunk_rows(d_model, z.ld, n_tokens, 1, 0, n_tokens)};
}

// What the forward makes besides its results. A training forward keeps all of it for the backward.
struct Kept {
  void *xs, *a1;                  // [L, D] permuted rows, [L, 2H] pre-activations (training only)
  void *logits, *w_all;           // [T, ld] unless the caller brought logits; [T, kS]
  int64_t* idx_all;
  int32_t *sorted_ids, *expert_ids, *pad_offsets, *counts_all, *n_post_pad, *inv_ids;
  void* router_wp;                // [D, ld]
  void *bias_in, *bias_out;       // [E + S, 2H], [E + S, D]: both weight stacks' biases
  void* bias_out_k;               // [ld, D]: the routed experts' b_out, rows past E zero
  size_t total;
};
struct Has {                      // the optional parts that the layout depends on
  bool train, logits_in, bias_in, bias_out;
};
Kept carve_kept(void* p, int64_t n_tokens, int32_t d_model, int32_t d_hidden, int32_t n_experts,
                int32_t n_shared, int32_t top_k, const Has& h) {
  const Sizes z = sizes(n_tokens, n_experts, n_shared, top_k);
  Carver c(p);
  Kept k{};
  if (h.train) {
    k.xs = c.take(size_t(z.l_cap) * d_model * 2);
    k.a1 = c.take(size_t(z.l_cap) * 2 * d_hidden * 2);
  }
  if (!h.logits_in) k.logits = c.take(size_t(n_tokens) * z.ld * 2);
  k.w_all = c.take(size_t(z.m) * 2);
  k.idx_all = static_cast<int64_t*>(c.take(size_t(z.m) * 8));
  k.sorted_ids = static_cast<int32_t*>(c.take(size_t(z.l_cap) * 4));
  k.expert_ids = static_cast<int32_t*>(c.take(size_t(z.l_cap / 128 + 1) * 4));
  k.pad_offsets = static_cast<int32_t*>(c.take(size_t(z.n_all + 1) * 4));
  k.counts_all = static_cast<int32_t*>(c.take(size_t(z.n_all) * 4));
  k.n_post_pad = static_cast<int32_t*>(c.take(4));
  k.inv_ids = static_cast<int32_t*>(c.take(size_t(z.m) * 4));
  k.router_wp = c.take(size_t(d_model) * z.ld * 2);
  if (h.bias_in) k.bias_in = c.take(size_t(z.n_all) * 2 * d_hidden * 2);
  if (h.bias_out) {
    k.bias_out = c.take(size_t(z.n_all) * d_model * 2);
    k.bias_out_k = c.take(size_t(z.ld) * d_model * 2);
  }
  k.total = c.used;
  return k;
}

// From this many tokens on the inference forward's GEMMs walk the tiles token window by token window instead
// of expert by expert (FinishArgs::order): a token's k rows are then gathered, and added to, while the token's
// row is in L2. 2048 tokens to a window.
constexpr int64_t ORDERED_TOKENS = 32768;
inline int32_t order_windows(int64_t n_tokens) {
  int32_t w = 1;
  while (w < 4096 && int64_t(w) * 2 * 2048 <= n_tokens) w *= 2;
  return w;
}

// Scratch of the forward: dead when it returns.
struct FwdScratch {
  void *hid, *y;                  // [L, H]; [L, D] (store combine only)
  void* block_hist;
  size_t block_hist_bytes;
  void* front;                    // of the router's front of a small batch
  int2* order;                    // [L / 128] the tiles' order (large batches only)
  float* colsum;
  size_t total;
};
FwdScratch carve_fwd(void* p, int64_t n_tokens, int32_t d_model, int32_t d_hidden,
                     int32_t n_experts, int32_t n_shared, int32_t top_k, bool store) {
  const Sizes z = sizes(n_tokens, n_experts, n_shared, top_k);
  Carver c(p);
  FwdScratch f{};
  f.hid = c.take(size_t(z.l_cap) * d_hidden * 2);
  f.block_hist_bytes = moe_b200_router_dispatch_scratch_bytes(n_tokens, z.n_all);
  f.block_hist = c.take(f.block_hist_bytes);
  f.front = c.take(moe::router_front_scratch_bytes(n_tokens, n_experts, n_shared));
  if (n_tokens >= ORDERED_TOKENS) f.order = static_cast<int2*>(c.take(size_t(z.l_cap / 128 + 1) * 8));
  f.colsum = static_cast<float*>(c.take(size_t(n_experts) * 4));
  if (store) f.y = c.take(size_t(z.l_cap) * d_model * 2);
  f.total = c.used;
  return f;
}

struct BwdScratch {
  void *douts, *da1, *hidw, *dtw, *dl, *d_router_padded, *part_in, *part_out, *part_r;
  void *ydx, *dx_router;          // store combine only
  void* b_extra;                  // [T, ld]: <dOut[t], b_out[e]> (with b_out only)
  float *db_in, *db_out;          // fp32 column sums (with biases only); one buffer
  size_t part_in_bytes, part_out_bytes, part_r_bytes, total;
};
int carve_bwd(void* p, int64_t n_tokens, int32_t d_model, int32_t d_hidden, int32_t n_experts,
              int32_t n_shared, int32_t top_k, bool store, bool bias_in, bool bias_out,
              BwdScratch* b) {
  const Sizes z = sizes(n_tokens, n_experts, n_shared, top_k);
  const Chunks ks = chunks_of(z, n_tokens, d_model, d_hidden);
  Carver c(p);
  *b = BwdScratch{};
  b->douts = c.take(size_t(z.l_cap) * d_model * 2);
  b->da1 = c.take(size_t(z.l_cap) * 2 * d_hidden * 2);
  b->hidw = c.take(size_t(z.l_cap) * d_hidden * 2);
  b->dtw = c.take(size_t(z.m) * 2);
  b->dl = c.take(size_t(n_tokens) * z.ld * 2);
  b->d_router_padded = c.take(size_t(d_model) * z.ld * 2);
  int rc = moe_b200_wgrad_scratch_bytes(d_model, 2 * d_hidden, z.l_cap, z.n_all, 1, ks.in,
                                        &b->part_in_bytes);
  if (rc != MOE_B200_OK) return rc;
  rc = moe_b200_wgrad_scratch_bytes(d_hidden, d_model, z.l_cap, z.n_all, 1, ks.out,
                                    &b->part_out_bytes);
  if (rc != MOE_B200_OK) return rc;
  rc = moe_b200_wgrad_scratch_bytes(d_model, z.ld, n_tokens, 1, 0, ks.router, &b->part_r_bytes);
  if (rc != MOE_B200_OK) return rc;
  b->part_in = c.take(b->part_in_bytes);
  b->part_out = c.take(b->part_out_bytes);
  b->part_r = c.take(b->part_r_bytes);
  if (store) {
    b->ydx = c.take(size_t(z.l_cap) * d_model * 2);
    b->dx_router = c.take(size_t(n_tokens) * d_model * 2);
  }
  if (bias_out) b->b_extra = c.take(size_t(n_tokens) * z.ld * 2);
  if (bias_in) b->db_in = static_cast<float*>(c.take(size_t(z.n_all) * 2 * d_hidden * 4));
  if (bias_out) b->db_out = static_cast<float*>(c.take(size_t(z.n_all) * d_model * 4));
  b->total = c.used;
  return MOE_B200_OK;
}

inline bool bad_shape(int64_t n_tokens, int32_t d_model, int32_t d_hidden, int32_t n_experts,
                      int32_t n_shared, int32_t top_k) {
  return n_tokens < 1 || d_model < 64 || d_hidden < 1 || n_experts < 1 || n_shared < 0 ||
         top_k < 1 || top_k > n_experts;
}

#define STEP(call)                   \
  do {                               \
    const int rc_ = (call);          \
    if (rc_ != MOE_B200_OK) return rc_; \
    ++launched;                      \
  } while (0)

// Everything a forward reads and writes, resolved to pointers. desc.router_w may be null when
// kept.router_wp already holds the padded weight.
struct Fwd {
  moe_b200_block_desc d;
  Kept k;
  FwdScratch s;
  void* out;
  float* aux;                     // null with counts: the caller wants neither
  int32_t aux_is_16bit;
  int32_t* counts;
  int64_t* dropped;
  bool train;
};

int run_forward(const Fwd& f, int32_t* n_launches, cudaStream_t st) {
  const moe_b200_block_desc& d = f.d;
  const Sizes z = sizes(d.n_tokens, d.n_experts, d.n_shared, d.top_k);
  const int64_t T = d.n_tokens;
  const int32_t D = d.d_model, H = d.d_hidden, E = d.n_experts, S = d.n_shared;
  void* stream = st;
  int launched = 0;
  const int32_t* first_shared = f.k.pad_offsets + E;   // start of the first shared run
  // a small batch's front end reads the router weight as it is and needs nothing prepared
  const bool front = !d.logits_in && d.router_w &&
                     moe::router_front_covers(T, D, E, S, d.top_k, d.x, d.router_w);
  float* colsum = d.full_softmax && !front ? f.s.colsum : nullptr;

  PrepArgs pa{};
  auto job = [&](const void* src, int32_t rows, int32_t cols, void* dst, int32_t dst_rows,
                 int32_t dst_ld) {
    pa.job[pa.n_jobs++] = PrepJob{static_cast<const uint16_t*>(src), static_cast<uint16_t*>(dst),
                                  src ? rows : 0, cols, dst_rows, dst_ld};
  };
  auto below = [](void* p, int64_t values) { return static_cast<uint16_t*>(p) + values; };
  if (d.router_w && !front) job(d.router_w, D, E, f.k.router_wp, D, z.ld);
  if (f.k.bias_in) {
    job(d.b_in, E, 2 * H, f.k.bias_in, E, 2 * H);
    if (S) job(d.b_sh_in, S, 2 * H, below(f.k.bias_in, int64_t(E) * 2 * H), S, 2 * H);
  }
  if (f.k.bias_out) {
    job(d.b_out, E, D, f.k.bias_out, E, D);
    if (S) job(d.b_sh_out, S, D, below(f.k.bias_out, int64_t(E) * D), S, D);
    job(d.b_out, E, D, f.k.bias_out_k, z.ld, D);
  }
  if (colsum) {
    pa.clear = colsum;
    pa.n_clear = E;
  }
  if (pa.n_jobs || pa.n_clear) STEP(prep(pa, st));

  int2* const order = f.train || !f.counts ? nullptr : f.s.order;
  const moe::FinishArgs fin{f.counts, colsum, f.aux, f.dropped, T, d.aux_coef, E, f.aux_is_16bit,
                            order, order_windows(T)};
  if (front) {
    const moe::ScatterArgs sc{f.k.counts_all, f.k.pad_offsets, f.k.n_post_pad, f.k.expert_ids,
                              z.l_cap / 128, f.k.inv_ids, d.capacity, E, fin};
    const moe::FrontCall fc{d.x, d.router_w, d.logit_bias, d.noise, T, D, E, S, d.top_k, d.normalize,
                            d.full_softmax, f.k.w_all, f.k.idx_all, f.train ? f.k.logits : nullptr,
                            f.train ? f.k.router_wp : nullptr, z.ld, f.k.sorted_ids, sc, f.s.front,
                            d.status};
    STEP(moe::router_front(fc, st));
    ++launched;
  } else {
    // router: logits GEMM against the padded weight (one fixed group, no pair weights), then
    // routing + dispatch
    const void* logits = d.logits_in ? d.logits_in : f.k.logits;
    const int32_t ld = d.logits_in ? E : z.ld;
    if (!d.logits_in)
      STEP(moe_b200_down_gemm(d.x, T, D, f.k.router_wp, 1, nullptr, 0, z.ld, nullptr, nullptr, 1,
                              nullptr, nullptr, 0, f.k.logits, nullptr, d.status, stream));
    int n_disp = 0;
    STEP(moe::router_dispatch(logits, ld, d.logit_bias, d.noise, T, E, d.top_k, S, d.normalize,
                              d.full_softmax, f.k.w_all, f.k.idx_all, colsum, f.k.sorted_ids,
                              f.k.expert_ids, f.k.pad_offsets, f.k.counts_all, f.k.n_post_pad,
                              f.k.inv_ids, f.s.block_hist, f.s.block_hist_bytes, d.capacity, fin, d.status,
                              stream, &n_disp));
    launched += n_disp - 1;
  }
  // experts: up/gate + GLU, gathering the token rows itself; a training forward leaves them in slot
  // order on the way, for the weight gradients
  if (f.train) {
    STEP(moe::up_gemm(d.x, z.l_cap, D, d.w_in, E, d.w_sh_in, S, H, f.k.expert_ids, f.k.n_post_pad, 0,
                      f.k.sorted_ids, z.ks, z.m, d.activation, f.s.hid, f.k.a1, S ? d.x : nullptr,
                      S ? T : 0, f.k.pad_offsets, f.k.bias_in, f.k.xs, nullptr, d.status, stream));
  } else {
    STEP(moe::up_gemm(d.x, z.l_cap, D, d.w_in, E, d.w_sh_in, S, H, f.k.expert_ids, f.k.n_post_pad, 0,
                      f.k.sorted_ids, z.ks, z.m, d.activation, f.s.hid, nullptr, S ? d.x : nullptr,
                      S ? T : 0, f.k.pad_offsets, f.k.bias_in, nullptr, order, d.status, stream));
  }
  // down + combine
  if (d.store_combine) {
    STEP(moe_b200_down_gemm(f.s.hid, z.l_cap, H, d.w_out, E, d.w_sh_out, S, D, f.k.expert_ids,
                            f.k.n_post_pad, 0, f.k.sorted_ids, f.k.w_all, z.m, f.s.y,
                            f.k.bias_out, d.status, stream));
    STEP(moe_b200_combine(f.s.y, f.k.inv_ids, T, z.ks, D, d.residual, nullptr, f.out, stream));
  } else if (S && !f.k.bias_out) {
    // the shared experts' share, and the residual, stored, are the accumulator's first value
    STEP(moe::down_gemm_sum(f.s.hid, z.l_cap, H, d.w_sh_out, S, D, first_shared, T, d.residual,
                            f.out, d.status, stream));
    STEP(moe::down_gemm_acc(f.s.hid, z.l_cap, H, d.w_out, E, nullptr, 0, D, f.k.expert_ids, first_shared, 0,
                            f.k.sorted_ids, f.k.w_all, z.m, z.ks, f.out, T, nullptr, order, d.status,
                            stream));
  } else {
    if (d.residual) STEP(copy_words(d.residual, f.out, T * D / 2, st));
    else STEP(zero_words(f.out, T * D / 2, st));
    STEP(moe::down_gemm_acc(f.s.hid, z.l_cap, H, d.w_out, E, d.w_sh_out, S, D, f.k.expert_ids,
                            f.k.n_post_pad, 0, f.k.sorted_ids, f.k.w_all, z.m, z.ks, f.out, T,
                            f.k.bias_out, order, d.status, stream));
  }
  if (n_launches) *n_launches = launched;
  return MOE_B200_OK;
}

struct Bwd {
  moe_b200_block_desc d;
  Kept k;
  BwdScratch s;
  const void* grad_out;
  const float* grad_aux;
  void *dx, *d_router, *dw_in, *dw_out, *dw_sh_in, *dw_sh_out, *db_in, *db_out;
  void *side_a, *side_b;
};

// The four events of the fork and the join. Sets are kept between calls, one per call in progress at
// once, and live as long as the process (there is no point at which a static could destroy them:
// the runtime may already be gone).
struct ForkEvents {
  cudaEvent_t fork = nullptr, dx = nullptr, a = nullptr, b = nullptr;
};
class ForkEventsLease {
 public:
  ForkEventsLease() {
    if (cudaGetDevice(&dev_) != cudaSuccess || dev_ < 0 || dev_ >= MAX_DEVICES) return;
    {
      std::lock_guard<std::mutex> lock(mutex());
      std::vector<ForkEvents>& pool = pools()[dev_];
      if (!pool.empty()) {
        ev = pool.back();
        pool.pop_back();
        ok = true;
        return;
      }
    }
    ok = true;
    for (cudaEvent_t* p : {&ev.fork, &ev.dx, &ev.a, &ev.b})
      ok = ok && cudaEventCreateWithFlags(p, cudaEventDisableTiming) == cudaSuccess;
  }
  ~ForkEventsLease() {
    if (!ok) return;
    std::lock_guard<std::mutex> lock(mutex());
    pools()[dev_].push_back(ev);
  }
  ForkEventsLease(const ForkEventsLease&) = delete;
  ForkEvents ev;
  bool ok = false;

 private:
  static constexpr int MAX_DEVICES = 64;
  static std::mutex& mutex() {
    static std::mutex* m = new std::mutex;
    return *m;
  }
  static std::vector<ForkEvents>* pools() {
    static std::vector<ForkEvents>* p = new std::vector<ForkEvents>[MAX_DEVICES];
    return p;
  }
  int dev_ = -1;
};

// From more tokens than this, dX adds the router's share itself (its weights' tiles as one more run). As a
// launch of its own on a side stream it finds no room beside dX's CTAs and comes after them: 16384 tokens
// 419 against 405 us with it in dX, 5000 graphed 231 against 229. But then dX has to wait for another
// stream and loses its early launch: 2048 graphed 163 against 168, 300 the same.
constexpr int64_t DX_WITH_ROUTER_TOKENS = 4096;

int run_backward(const Bwd& b, int32_t* n_launches, cudaStream_t main_st) {
  const moe_b200_block_desc& d = b.d;
  const Sizes z = sizes(d.n_tokens, d.n_experts, d.n_shared, d.top_k);
  const int64_t T = d.n_tokens;
  const int32_t D = d.d_model, H = d.d_hidden, E = d.n_experts, S = d.n_shared;
  void* stream = main_st;
  // the two side branches run on the caller's side streams, or in line when none are given
  cudaStream_t sa = b.side_a ? static_cast<cudaStream_t>(b.side_a) : main_st;
  cudaStream_t sb = b.side_b ? static_cast<cudaStream_t>(b.side_b) : main_st;
  int launched = 0;
  const int32_t* first_shared = b.k.pad_offsets + E;
  const int32_t* live = S ? first_shared : b.k.n_post_pad;
  const bool store = d.store_combine != 0;
  const int64_t longest = longest_run(T);
  const Chunks ks = chunks_of(z, T, D, H);
  const int32_t* offs = S ? b.k.pad_offsets : nullptr;

  STEP(moe::dhidden_glu_bwd(b.grad_out, z.l_cap, D, d.w_out, E, d.w_sh_out, S, H, b.k.expert_ids,
                            b.k.n_post_pad, 0, b.k.sorted_ids, z.ks, b.k.w_all, z.m, b.k.a1,
                            d.activation, b.s.da1, b.s.hidw, b.s.dtw, S ? b.grad_out : nullptr,
                            S ? T : 0, offs, b.s.douts, d.status, stream));
  // fork: everything below depends only on the launch above
  const ForkEventsLease lease;
  if (!lease.ok) return MOE_B200_ERR_CUDA;
  const ForkEvents* ev = &lease.ev;
#define CU(call) \
  if ((call) != cudaSuccess) return MOE_B200_ERR_CUDA
  CU(cudaEventRecord(ev->fork, main_st));
  if (sa != main_st) CU(cudaStreamWaitEvent(sa, ev->fork, 0));
  if (sb != main_st) CU(cudaStreamWaitEvent(sb, ev->fork, 0));

  // main: dx's first value (the shared experts' share, stored), dW_in, the routed rows of dx. The router's
  // share of dx comes with those (dx_with_router) or by a launch of its own on side b.
  const bool dx_with_router = !store && T > DX_WITH_ROUTER_TOKENS;
  if (!store) {
    if (S)
      STEP(moe_b200_dx_gemm_sum(b.s.da1, z.l_cap, H, d.w_sh_in, S, D, first_shared, T, b.dx,
                                d.status, stream));
    else
      STEP(zero_words(b.dx, T * D / 2, main_st));
    if (!dx_with_router) CU(cudaEventRecord(ev->dx, main_st));
  }
  STEP(moe::wgrad(b.k.xs, 0, D, b.s.da1, 0, 2 * H, z.l_cap, b.k.pad_offsets, z.n_all, ks.in, nullptr, 0,
                  0, 0, b.dw_in, E, S ? b.dw_sh_in : nullptr, b.s.part_in, b.s.part_in_bytes,
                  S ? d.x : nullptr, S ? T : 0, S ? 1 : 0, longest, 2 * H, d.status, stream));
  // side a: dW_out, then the bias gradients (column sums over the runs)
  STEP(moe::wgrad(b.s.hidw, 0, H, b.s.douts, 0, D, z.l_cap, b.k.pad_offsets, z.n_all, ks.out, nullptr, 0,
                  0, 0, b.dw_out, E, S ? b.dw_sh_out : nullptr, b.s.part_out, b.s.part_out_bytes,
                  S ? b.grad_out : nullptr, S ? T : 0, S ? 2 : 0, longest, D, d.status, sa));
  // side b: the router's backward. With b_out a pair's d(topk_w) gains <dOut[t], b_out[e]>: one row GEMM
  // dOut @ b_out^T over all experts, read at the pair's column by the router kernel.
  if (b.s.b_extra)
    STEP(moe_b200_dx_gemm(b.grad_out, T, D / 2, b.k.bias_out_k, 1, nullptr, 0, z.ld, nullptr,
                          nullptr, 1, b.s.b_extra, d.status, sb));
  STEP(moe::router_fused_bwd(d.logits_in ? d.logits_in : b.k.logits, d.logits_in ? E : z.ld,
                             d.logit_bias, d.noise, b.k.idx_all, b.s.dtw, b.s.b_extra, z.ld,
                             d.capacity > 0 ? b.k.inv_ids : nullptr, T, E, d.top_k, S,
                             d.normalize, d.full_softmax, b.grad_aux, b.k.counts_all, d.aux_coef,
                             b.s.dl, z.ld, sb));
  if (dx_with_router && sb != main_st) CU(cudaEventRecord(ev->dx, sb));
  if (store) {
    STEP(moe_b200_dx_gemm(b.s.da1, z.l_cap, H, d.w_in, E, d.w_sh_in, S, D, b.k.expert_ids,
                          b.k.n_post_pad, 0, b.s.ydx, d.status, stream));
  } else {
    if (dx_with_router && sb != main_st) CU(cudaStreamWaitEvent(main_st, ev->dx, 0));
    STEP(moe::dx_gemm_acc(b.s.da1, z.l_cap, H, d.w_in, E, nullptr, 0, D, b.k.expert_ids, live, 0,
                          b.k.sorted_ids, z.m, z.ks, b.dx, T, b.k.pad_offsets,
                          dx_with_router ? b.s.dl : nullptr, b.k.router_wp, z.ld, d.status, stream));
  }
  const int32_t n_bi = b.s.db_in ? z.n_all * 2 * H : 0, n_bo = b.s.db_out ? z.n_all * D : 0;
  if (n_bi) {
    STEP(zero_words(b.s.db_in, n_bi, sa));
    STEP(moe_b200_segment_colsum(b.s.da1, z.l_cap, 2 * H, b.k.expert_ids, b.k.n_post_pad, nullptr,
                                 z.n_all, nullptr, nullptr, 0, nullptr, 0, 0, b.s.db_in, sa));
    STEP(to_bf16(b.s.db_in, b.db_in, n_bi, sa));
  }
  if (n_bo) {
    STEP(zero_words(b.s.db_out, n_bo, sa));
    STEP(moe_b200_segment_colsum(b.s.douts, z.l_cap, D, b.k.expert_ids, b.k.n_post_pad, offs,
                                 z.n_all, b.k.sorted_ids, b.k.w_all, z.m,
                                 S ? b.grad_out : nullptr, S ? T : 0, E, b.s.db_out, sa));
    STEP(to_bf16(b.s.db_out, b.db_out, n_bo, sa));
  }
  // side b: the router's weight gradient (a product of one chunk is stored with the padded width and
  // copied), and its share of dx: as rows of their own with a stored combine, or added
  const bool padded = E != z.ld && T <= ks.router;
  STEP(moe::wgrad(d.x, 0, D, b.s.dl, 0, z.ld, T, nullptr, 1, ks.router, nullptr, 0, 0, 0,
                  padded ? b.s.d_router_padded : b.d_router, 1, nullptr, b.s.part_r,
                  b.s.part_r_bytes, nullptr, 0, 0, T, padded ? z.ld : E, d.status, sb));
  if (padded) STEP(moe_b200_copy_cols(b.s.d_router_padded, D, E, z.ld, b.d_router, E, sb));
  if (store) {
    STEP(moe_b200_dx_gemm(b.s.dl, T, z.ld / 2, b.k.router_wp, 1, nullptr, 0, D, nullptr, nullptr,
                          1, b.s.dx_router, d.status, sb));
  } else if (!dx_with_router) {
    if (sb != main_st) CU(cudaStreamWaitEvent(sb, ev->dx, 0));
    STEP(moe_b200_dx_gemm_acc(b.s.dl, T, z.ld / 2, b.k.router_wp, 1, nullptr, 0, D, nullptr,
                              nullptr, 1, nullptr, 0, 1, b.dx, T, nullptr, d.status, sb));
  }
  // join
  if (sa != main_st) {
    CU(cudaEventRecord(ev->a, sa));
    CU(cudaStreamWaitEvent(main_st, ev->a, 0));
  }
  if (sb != main_st) {
    CU(cudaEventRecord(ev->b, sb));
    CU(cudaStreamWaitEvent(main_st, ev->b, 0));
  }
#undef CU
  if (store)
    STEP(moe_b200_combine(b.s.ydx, b.k.inv_ids, T, z.ks, D, b.s.dx_router, nullptr, b.dx, stream));
  // the weight gradients' reduction passes
  launched += (longest > ks.in) + (longest > ks.out) + (T > ks.router);
  if (n_launches) *n_launches = launched;
  return MOE_B200_OK;
}

// The checks every descriptor call makes before it touches a pointer.
int check_desc(const moe_b200_block_desc* d) {
  if (d == nullptr) return MOE_B200_ERR_NULL;
  if (bad_shape(d->n_tokens, d->d_model, d->d_hidden, d->n_experts, d->n_shared, d->top_k) ||
      d->capacity < 0)
    return MOE_B200_ERR_SHAPE;
  return MOE_B200_OK;
}
inline Has has_of(const moe_b200_block_desc* d, bool train) {
  return Has{train, d->logits_in != nullptr, d->b_in || d->b_sh_in, d->b_out || d->b_sh_out};
}
inline Kept kept_of(const moe_b200_block_desc* d, void* p, bool train) {
  return carve_kept(p, d->n_tokens, d->d_model, d->d_hidden, d->n_experts, d->n_shared, d->top_k,
                    has_of(d, train));
}

}  // namespace

extern "C" {

size_t moe_b200_block_kept_bytes(const moe_b200_block_desc* d, int32_t train) {
  if (check_desc(d) != MOE_B200_OK) return 0;
  return kept_of(d, nullptr, train != 0).total;
}

size_t moe_b200_block_forward_scratch_bytes(const moe_b200_block_desc* d) {
  if (check_desc(d) != MOE_B200_OK) return 0;
  return carve_fwd(nullptr, d->n_tokens, d->d_model, d->d_hidden, d->n_experts, d->n_shared,
                   d->top_k, d->store_combine != 0).total;
}

size_t moe_b200_block_backward_scratch_bytes(const moe_b200_block_desc* d) {
  if (check_desc(d) != MOE_B200_OK) return 0;
  BwdScratch b;
  const Has h = has_of(d, true);
  if (carve_bwd(nullptr, d->n_tokens, d->d_model, d->d_hidden, d->n_experts, d->n_shared, d->top_k,
                d->store_combine != 0, h.bias_in, h.bias_out, &b) != MOE_B200_OK)
    return 0;
  return b.total;
}

int moe_b200_block_forward(const moe_b200_block_desc* d, int32_t train, void* out, void* aux,
                           int32_t aux_is_16bit, int32_t* counts, int64_t* dropped, void* kept,
                           size_t kept_bytes, void* scratch, size_t scratch_bytes,
                           int32_t* n_launches, void* stream) {
  const int rc = check_desc(d);
  if (rc != MOE_B200_OK) return rc;
  if (!d->x || !d->router_w || !d->w_in || !d->w_out || !d->status || !out || !aux || !counts ||
      !kept || !scratch)
    return MOE_B200_ERR_NULL;
  if (d->n_shared > 0 && (!d->w_sh_in || !d->w_sh_out)) return MOE_B200_ERR_NULL;
  if (kept_bytes < moe_b200_block_kept_bytes(d, train) ||
      scratch_bytes < moe_b200_block_forward_scratch_bytes(d))
    return MOE_B200_ERR_SCRATCH;
  Fwd f{};
  f.d = *d;
  f.train = train != 0;
  f.k = kept_of(d, kept, f.train);
  f.s = carve_fwd(scratch, d->n_tokens, d->d_model, d->d_hidden, d->n_experts, d->n_shared,
                  d->top_k, d->store_combine != 0);
  f.out = out;
  f.aux = static_cast<float*>(aux);
  f.aux_is_16bit = aux_is_16bit && !d->full_softmax;
  f.counts = counts;
  f.dropped = dropped;
  return run_forward(f, n_launches, static_cast<cudaStream_t>(stream));
}

int moe_b200_block_backward(const moe_b200_block_desc* d, const void* grad_out,
                            const float* grad_aux, const void* kept, size_t kept_bytes, void* dx,
                            void* d_router, void* dw_in, void* dw_out, void* dw_sh_in,
                            void* dw_sh_out, void* db_in, void* db_out, void* scratch,
                            size_t scratch_bytes, void* side_stream_a, void* side_stream_b,
                            int32_t* n_launches, void* stream) {
  const int rc = check_desc(d);
  if (rc != MOE_B200_OK) return rc;
  if (!d->x || !d->w_in || !d->w_out || !d->status || !grad_out || !kept || !dx || !d_router ||
      !dw_in || !dw_out || !scratch)
    return MOE_B200_ERR_NULL;
  if (d->n_shared > 0 && (!d->w_sh_in || !d->w_sh_out || !dw_sh_in || !dw_sh_out))
    return MOE_B200_ERR_NULL;
  const Has h = has_of(d, true);
  if ((h.bias_in && !db_in) || (h.bias_out && !db_out)) return MOE_B200_ERR_NULL;
  if (kept_bytes < moe_b200_block_kept_bytes(d, 1)) return MOE_B200_ERR_SCRATCH;
  Bwd b{};
  b.d = *d;
  b.k = kept_of(d, const_cast<void*>(kept), true);
  const int rcb = carve_bwd(scratch, d->n_tokens, d->d_model, d->d_hidden, d->n_experts,
                            d->n_shared, d->top_k, d->store_combine != 0, h.bias_in, h.bias_out,
                            &b.s);
  if (rcb != MOE_B200_OK) return rcb;
  if (scratch_bytes < b.s.total) return MOE_B200_ERR_SCRATCH;
  b.grad_out = grad_out;
  b.grad_aux = grad_aux;
  b.dx = dx;
  b.d_router = d_router;
  b.dw_in = dw_in;
  b.dw_out = dw_out;
  b.dw_sh_in = dw_sh_in;
  b.dw_sh_out = dw_sh_out;
  b.db_in = db_in;
  b.db_out = db_out;
  b.side_a = side_stream_a;
  b.side_b = side_stream_b;
  return run_backward(b, n_launches, static_cast<cudaStream_t>(stream));
}

// The same sequences for hosts that hold every kept tensor as a buffer of its own.
static moe_b200_block_desc plain_desc(const void* x, int64_t n_tokens, int32_t d_model,
                                      const void* w_in, const void* w_out, int32_t n_experts,
                                      int32_t d_hidden, const void* w_sh_in, const void* w_sh_out,
                                      int32_t n_shared, int32_t top_k, int32_t normalize,
                                      int32_t activation, const float* logit_bias,
                                      int32_t* status) {
  moe_b200_block_desc d{};
  d.n_tokens = n_tokens;
  d.d_model = d_model;
  d.d_hidden = d_hidden;
  d.n_experts = n_experts;
  d.n_shared = n_shared;
  d.top_k = top_k;
  d.normalize = normalize;
  d.activation = activation;
  d.x = x;
  d.w_in = w_in;
  d.w_out = w_out;
  d.w_sh_in = w_sh_in;
  d.w_sh_out = w_sh_out;
  d.logit_bias = logit_bias;
  d.status = status;
  return d;
}

size_t moe_b200_block_fwd_scratch_bytes(int64_t n_tokens, int32_t d_model, int32_t d_hidden,
                                        int32_t n_experts, int32_t n_shared, int32_t top_k) {
  if (bad_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k)) return 0;
  return carve_fwd(nullptr, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, false).total;
}

size_t moe_b200_block_infer_scratch_bytes(int64_t n_tokens, int32_t d_model, int32_t d_hidden,
                                          int32_t n_experts, int32_t n_shared, int32_t top_k) {
  if (bad_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k)) return 0;
  return carve_kept(nullptr, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, Has{}).total +
         carve_fwd(nullptr, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, true).total;
}

size_t moe_b200_block_bwd_scratch_bytes(int64_t n_tokens, int32_t d_model, int32_t d_hidden,
                                        int32_t n_experts, int32_t n_shared, int32_t top_k) {
  if (bad_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k)) return 0;
  BwdScratch b;
  if (carve_bwd(nullptr, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, false, false,
                false, &b) != MOE_B200_OK)
    return 0;
  return b.total;
}

int moe_b200_block_infer(const void* x, int64_t n_tokens, int32_t d_model,
                         const void* router_w_padded, const float* logit_bias, const void* w_in,
                         const void* w_out, int32_t n_experts, int32_t d_hidden,
                         const void* w_sh_in, const void* w_sh_out, int32_t n_shared,
                         int32_t top_k, int32_t normalize, int32_t activation,
                         const void* residual, int32_t atomic_combine, void* out, void* scratch,
                         size_t scratch_bytes, int32_t* n_launches, int32_t* status,
                         void* stream) {
  if (bad_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k)) return MOE_B200_ERR_SHAPE;
  if (!x || !router_w_padded || !w_in || !w_out || !out || !scratch || !status)
    return MOE_B200_ERR_NULL;
  if (n_shared > 0 && (!w_sh_in || !w_sh_out)) return MOE_B200_ERR_NULL;
  if (scratch_bytes < moe_b200_block_infer_scratch_bytes(n_tokens, d_model, d_hidden, n_experts,
                                                         n_shared, top_k))
    return MOE_B200_ERR_SCRATCH;
  Fwd f{};
  f.d = plain_desc(x, n_tokens, d_model, w_in, w_out, n_experts, d_hidden, w_sh_in, w_sh_out,
                   n_shared, top_k, normalize, activation, logit_bias, status);
  f.d.residual = residual;
  f.d.store_combine = !atomic_combine;
  f.k = carve_kept(scratch, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, Has{});
  f.s = carve_fwd(static_cast<char*>(scratch) + f.k.total, n_tokens, d_model, d_hidden, n_experts,
                  n_shared, top_k, true);
  f.k.router_wp = const_cast<void*>(router_w_padded);
  f.out = out;
  return run_forward(f, n_launches, static_cast<cudaStream_t>(stream));
}

int moe_b200_block_fwd(const void* x, int64_t n_tokens, int32_t d_model, const void* router_w,
                       const float* logit_bias, const float* noise, const void* w_in,
                       const void* w_out, int32_t n_experts, int32_t d_hidden,
                       const void* w_sh_in, const void* w_sh_out, int32_t n_shared,
                       int32_t top_k, int32_t normalize, int32_t full_softmax, float aux_coef,
                       int32_t activation, void* out, float* aux, int32_t* counts, void* xs,
                       void* a1, void* logits, void* w_all, int64_t* idx_all,
                       int32_t* sorted_ids, int32_t* expert_ids, int32_t* pad_offsets,
                       int32_t* counts_all, int32_t* n_post_pad, int32_t* inv_ids,
                       void* router_w_padded, void* scratch, size_t scratch_bytes,
                       int32_t* n_launches, int32_t* status, void* stream) {
  if (bad_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k)) return MOE_B200_ERR_SHAPE;
  if (!x || !router_w || !w_in || !w_out || !out || !aux || !counts || !xs || !a1 || !logits ||
      !w_all || !idx_all || !sorted_ids || !expert_ids || !pad_offsets || !counts_all ||
      !n_post_pad || !inv_ids || !router_w_padded || !scratch || !status)
    return MOE_B200_ERR_NULL;
  if (n_shared > 0 && (!w_sh_in || !w_sh_out)) return MOE_B200_ERR_NULL;
  Fwd f{};
  f.s = carve_fwd(scratch, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, false);
  if (scratch_bytes < f.s.total) return MOE_B200_ERR_SCRATCH;
  f.d = plain_desc(x, n_tokens, d_model, w_in, w_out, n_experts, d_hidden, w_sh_in, w_sh_out,
                   n_shared, top_k, normalize, activation, logit_bias, status);
  f.d.router_w = router_w;
  f.d.noise = noise;
  f.d.full_softmax = full_softmax;
  f.d.aux_coef = aux_coef;
  f.train = true;
  f.k.xs = xs;
  f.k.a1 = a1;
  f.k.logits = logits;
  f.k.w_all = w_all;
  f.k.idx_all = idx_all;
  f.k.sorted_ids = sorted_ids;
  f.k.expert_ids = expert_ids;
  f.k.pad_offsets = pad_offsets;
  f.k.counts_all = counts_all;
  f.k.n_post_pad = n_post_pad;
  f.k.inv_ids = inv_ids;
  f.k.router_wp = router_w_padded;
  f.out = out;
  f.aux = aux;
  f.counts = counts;
  return run_forward(f, n_launches, static_cast<cudaStream_t>(stream));
}

int moe_b200_block_bwd(const void* grad_out, const float* grad_aux, const void* x,
                       int64_t n_tokens, int32_t d_model, const float* logit_bias,
                       const float* noise, const void* w_in, const void* w_out,
                       int32_t n_experts, int32_t d_hidden, const void* w_sh_in,
                       const void* w_sh_out, int32_t n_shared, int32_t top_k, int32_t normalize,
                       int32_t full_softmax, float aux_coef, int32_t activation, const void* xs,
                       const void* a1, const void* logits, const void* w_all,
                       const int64_t* idx_all, const int32_t* sorted_ids,
                       const int32_t* expert_ids, const int32_t* pad_offsets,
                       const int32_t* counts_all, const int32_t* n_post_pad,
                       const void* router_w_padded, void* dx, void* d_router, void* dw_in,
                       void* dw_out, void* dw_sh_in, void* dw_sh_out, void* scratch,
                       size_t scratch_bytes, void* side_stream_a, void* side_stream_b,
                       int32_t* n_launches, int32_t* status, void* stream) {
  if (bad_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k)) return MOE_B200_ERR_SHAPE;
  if (!grad_out || !x || !w_in || !w_out || !xs || !a1 || !logits || !w_all || !idx_all ||
      !sorted_ids || !expert_ids || !pad_offsets || !counts_all || !n_post_pad ||
      !router_w_padded || !dx || !d_router || !dw_in || !dw_out || !scratch || !status)
    return MOE_B200_ERR_NULL;
  if (n_shared > 0 && (!w_sh_in || !w_sh_out || !dw_sh_in || !dw_sh_out)) return MOE_B200_ERR_NULL;
  Bwd b{};
  const int rcb = carve_bwd(scratch, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k,
                            false, false, false, &b.s);
  if (rcb != MOE_B200_OK) return rcb;
  if (scratch_bytes < b.s.total) return MOE_B200_ERR_SCRATCH;
  b.d = plain_desc(x, n_tokens, d_model, w_in, w_out, n_experts, d_hidden, w_sh_in, w_sh_out,
                   n_shared, top_k, normalize, activation, logit_bias, status);
  b.d.noise = noise;
  b.d.full_softmax = full_softmax;
  b.d.aux_coef = aux_coef;
  b.k.xs = const_cast<void*>(xs);
  b.k.a1 = const_cast<void*>(a1);
  b.k.logits = const_cast<void*>(logits);
  b.k.w_all = const_cast<void*>(w_all);
  b.k.idx_all = const_cast<int64_t*>(idx_all);
  b.k.sorted_ids = const_cast<int32_t*>(sorted_ids);
  b.k.expert_ids = const_cast<int32_t*>(expert_ids);
  b.k.pad_offsets = const_cast<int32_t*>(pad_offsets);
  b.k.counts_all = const_cast<int32_t*>(counts_all);
  b.k.n_post_pad = const_cast<int32_t*>(n_post_pad);
  b.k.router_wp = const_cast<void*>(router_w_padded);
  b.grad_out = grad_out;
  b.grad_aux = grad_aux;
  b.dx = dx;
  b.d_router = d_router;
  b.dw_in = dw_in;
  b.dw_out = dw_out;
  b.dw_sh_in = dw_sh_in;
  b.dw_sh_out = dw_sh_out;
  b.side_a = side_stream_a;
  b.side_b = side_stream_b;
  return run_backward(b, n_launches, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
