// The router's front of a small batch (up to 2048 tokens) in two launches: logits, selection and the first
// pass of the dispatch by one kernel, plan and scatter by another. At these sizes the front is a chain of
// latencies, and the four launches of larger batches (router weight padded 2.5 us, logits GEMM 5.4, top-k
// and dispatch as one cluster 15.9) spend most of theirs apart from the work: three CTAs for 300 tokens,
// each with 128 tokens' selections (2.9 us of instruction issue on one SM) and half a dozen grid-wide or
// cluster-wide hand-overs.
//
// Here a CTA takes 16 tokens, so that 128 CTAs share 2048. It brings their rows and the whole router weight
// (as it is: [D, E], no padding pass) into shared memory, forms the logits with one tcgen05 accumulator and
// routes them from there. The M = 128 tile is 16 rows of tokens and 112 of whatever follows them in shared
// memory: rows are independent, and the tile costs 0.8 us however full it is. The products run in the order
// of the logits GEMM (K steps of 16), so the logits are the same bits.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/moe_b200.h"
#include "dispatch_scatter.cuh"
#include "gemm.cuh"
#include "per_device.cuh"
#include "route_token.cuh"
#include "routing.cuh"

namespace moe {

constexpr int FRONT_TOKENS = 16;
constexpr int FRONT_MAX_BLOCKS = 128;
constexpr int FRONT_THREADS = 512;
constexpr int FRONT_MAX_SMEM = 210 * 1024;   // beside the static part

struct FrontArgs {
  const __nv_bfloat16 *x, *w;     // [T, D], [D, E]
  const float* bias;              // [E] or null
  RouteArgs route;
  int64_t n_tokens;
  int32_t d_model;
  __nv_bfloat16* logits;          // [T, ld] or null
  __nv_bfloat16* w_padded;        // [D, ld] or null: the router weight with zeros past E, for the backward
  int32_t ld;
  int32_t* block_hist;            // [E + S][blocks]
  float* block_colsum;            // [E][blocks] or null
  int32_t* sorted_ids;            // [l_cap], painted with the sentinel
  int64_t l_cap;
  int32_t* status;
};

// Shared memory: rows [K / 64][16][64] and the weight [N / 64][K][64], both in the 128-byte swizzle
// (K-major and MN-major operands), then the logits [16][E] with rows of FRONT_LOGIT_LD.
constexpr int FRONT_LOGIT_LD = 132;   // values; rows 264 bytes apart: 8-byte reads without conflicts
struct FrontSmem {
  int w, box, logits, total;
};
__host__ __device__ __forceinline__ FrontSmem front_smem(int d_model, int n_experts) {
  FrontSmem s;
  s.w = (d_model + 63) / 64 * 2048;
  s.box = d_model * 128;
  s.logits = s.w + (n_experts + 63) / 64 * s.box;
  s.total = s.logits + FRONT_TOKENS * FRONT_LOGIT_LD * 2;
  if (s.total < s.w + 14336) s.total = s.w + 14336;   // what the M = 128 tile of the last K block reads
  s.total += 1024;                                    // (for the alignment)
  return s;
}

// NS: ceil(E / 32); epl: experts per lane of the four-lane form.
template <int NS>
__global__ void __launch_bounds__(FRONT_THREADS, 1) router_front_kernel(const FrontArgs p, int epl) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t mma_done;
  __shared__ uint32_t tmem_slot;
  __shared__ int32_t hist[MAX_EXPERTS];
  __shared__ float probs[FRONT_TOKENS][NS * 32], tmp[FRONT_TOKENS][RF4_MAX_TOPK];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int D = p.d_model, E = p.route.n_experts;
  const FrontSmem L = front_smem(D, E);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t t0 = int64_t(blockIdx.x) * FRONT_TOKENS;
  const int here = int(min(int64_t(FRONT_TOKENS), p.n_tokens - t0));
  if (tid == 0) {
    mbar_init(&mma_done, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 128);
    tmem_relinquish();
    pdl_trigger();
  }
  for (int e = tid; e < E + p.route.n_shared; e += FRONT_THREADS) hist[e] = 0;
  pdl_wait();

  // rows of 16-byte pieces; a weight row of E / 4 8-byte pieces, of which a thread copies one in every
  // `rows` rows
  const uint32_t a_u = smem_u32(smem), w_u = a_u + L.w;
  const int pieces = D / 8;
  for (int i = tid; i < FRONT_TOKENS * pieces; i += FRONT_THREADS) {
    const int r = i / pieces, c = i - r * pieces;
    cp_async_16(a_u + (c >> 3) * 2048 + r * 128 + (((c & 7) ^ (r & 7)) << 4),
                p.x + (r < here ? (t0 + r) * D + c * 8 : 0), r < here ? 16u : 0u);
  }
  const int quads = E / 4, rows = FRONT_THREADS / quads;
  const int k0 = tid / quads, n0 = 4 * (tid - k0 * quads);
  if (k0 < rows) {
    const uint32_t col = w_u + (n0 >> 6) * L.box + (n0 & 4) * 2, c = (n0 & 63) >> 3;
    const __nv_bfloat16* src = p.w + k0 * E + n0;
#pragma unroll 4
    for (int k = k0; k < D; k += rows, src += rows * E) cp_async_8(col + k * 128 + ((c ^ (k & 7)) << 4), src);
  }
  cp_async_wait_all();
  fence_proxy_async();       // (the tensor core reads through the async proxy)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (tid == 0) {
    const uint32_t idesc = umma_idesc(128, 0, false, true) | uint32_t((E + 15) / 16 * 2) << 17;
#pragma unroll 4
    for (int k = 0; k < D / 16; ++k)
      umma_f16(tmem, umma_desc(a_u + (k >> 2) * 2048 + (k & 3) * 32, 16, 1024),
               umma_desc(w_u + k * 2048, uint32_t(L.box), 1024), idesc, k ? 1u : 0u);
    umma_commit(&mma_done);
  }
  // Beside the MMAs: the sentinel fill (each block an equal slice) and the padded weight.
  const int kS = p.route.top_k + p.route.n_shared;
  const int32_t n_pairs = int32_t(p.n_tokens * kS);
  {
    const int64_t per = (p.l_cap + gridDim.x - 1) / gridDim.x, lo = per * blockIdx.x;
    const int64_t hi = min(lo + per, p.l_cap);
    for (int64_t i = lo + tid; i < hi; i += FRONT_THREADS) p.sorted_ids[i] = n_pairs;
  }
  if (p.w_padded != nullptr) {
    const int quads_out = p.ld / 4, rows = (D + gridDim.x - 1) / gridDim.x;
    const int k_lo = rows * blockIdx.x, k_hi = min(k_lo + rows, D);
    for (int i = k_lo * quads_out + tid; i < k_hi * quads_out; i += FRONT_THREADS) {
      const int k = i / quads_out, n = 4 * (i - k * quads_out);
      uint2 v = make_uint2(0u, 0u);
      if (n < E)
        v = *reinterpret_cast<const uint2*>(smem + L.w + (n >> 6) * L.box + k * 128 +
                                            ((((n & 63) >> 3) ^ (k & 7)) << 4) + (n & 4) * 2);
      *reinterpret_cast<uint2*>(p.w_padded + int64_t(k) * p.ld + n) = v;
    }
  }
  // accumulator -> bf16 logits; a warp of the first lane quadrant per 32 columns (lanes 0..15: tokens)
  __nv_bfloat16* lg = reinterpret_cast<__nv_bfloat16*>(smem + L.logits);
  if (!mbar_wait(&mma_done, 0, p.status)) atomicExch(p.status, ST_WAIT_TIMEOUT);
  tc_fence_after();
  if ((warp & 3) == 0 && warp * 8 < E) {
    float v[32];
    tmem_ld32(tmem + warp * 8, v);
    tmem_ld_wait();
    if (lane < FRONT_TOKENS)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v[4 * i], v[4 * i + 1]);
        const __nv_bfloat162 hi = __floats2bfloat162_rn(v[4 * i + 2], v[4 * i + 3]);
        *reinterpret_cast<uint2*>(lg + lane * FRONT_LOGIT_LD + warp * 8 + 4 * i) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 128);

  if (warp < here)   // a warp per token
    route_warp<NS>(p.route, lg + warp * FRONT_LOGIT_LD, p.bias, t0 + warp, epl, probs[warp], tmp[warp], hist);
  if (p.logits != nullptr) {
    const int quads_out = p.ld / 4;
    for (int i = tid; i < here * quads_out; i += FRONT_THREADS) {
      const int r = i / quads_out, n = 4 * (i - r * quads_out);
      *reinterpret_cast<uint2*>(p.logits + (t0 + r) * p.ld + n) =
          n < E ? *reinterpret_cast<const uint2*>(lg + r * FRONT_LOGIT_LD + n) : make_uint2(0u, 0u);
    }
  }
  __syncthreads();
  for (int e = tid; e < E + p.route.n_shared; e += FRONT_THREADS) {   // (every token visits the shared experts)
    p.block_hist[e * int(gridDim.x) + blockIdx.x] = e < E ? hist[e] : here;
    if (p.block_colsum != nullptr && e < E) {
      float s = 0.f;
      for (int r = 0; r < here; ++r) s += probs[r][e];
      p.block_colsum[e * int(gridDim.x) + blockIdx.x] = s;
    }
  }
}

// Plan and scatter behind the kernel above: dispatch_scatter_body's results for chunks of at most one pair
// per thread. Every global load is on its way before the first is used (a pair's expert beside the
// histogram table), the ranks inside the block are made under the plan, and two barriers remain.
__global__ void __launch_bounds__(FRONT_THREADS)
    router_front_scatter_kernel(const int64_t* idx_all, int32_t n_pairs, int n_experts,
                                int chunk, const int32_t* block_hist,
                                const float* block_colsum, int32_t* sorted_ids,
                                const ScatterArgs sc) {
  constexpr int WARPS = FRONT_THREADS / 32, MAX_WARPS = FRONT_TOKENS * 32 / 32;
  pdl_trigger();
  __shared__ int32_t total[MAX_EXPERTS], before[MAX_EXPERTS], off[MAX_EXPERTS + 1];
  __shared__ uint16_t mine[MAX_WARPS][MAX_EXPERTS];   // pairs of an expert in each warp of the block
  __shared__ float colsum[MAX_EXPERTS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, blk = int(blockIdx.x);
  const int n_blocks = int(gridDim.x);
  const int warps = (chunk + 31) / 32;
  for (int i = tid; i < warps * (MAX_EXPERTS / 2); i += FRONT_THREADS)
    reinterpret_cast<uint32_t*>(mine)[i] = 0u;
  __syncthreads();   // (a warp counts into its row below; ahead of the wait the barrier costs nothing)
  pdl_wait();
  const int64_t pair = int64_t(blk) * chunk + tid;
  const bool live_pair = tid < chunk && pair < n_pairs;
  const int e_mine = live_pair ? int(ld_prev(reinterpret_cast<const long long*>(idx_all) + pair)) : -1;
  const bool finish = sc.fin.counts != nullptr && blk == 0;
  constexpr int U = 6;   // experts of a warp at a time
  for (int e0 = warp; e0 < n_experts; e0 += U * WARPS) {
    int32_t v[U][4];
    float f[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = e0 + u * WARPS, b = lane + 32 * j;
        v[u][j] = e < n_experts && b < n_blocks ? ld_prev(block_hist + e * n_blocks + b) : 0;
        f[u][j] = finish && block_colsum != nullptr && e < sc.fin.n_experts && b < n_blocks
                      ? ld_prev(block_colsum + e * n_blocks + b)
                      : 0.f;
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * WARPS;
      int32_t bef = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (lane + 32 * j < blk) bef += v[u][j];
      const int32_t tot = __reduce_add_sync(0xffffffffu, v[u][0] + v[u][1] + v[u][2] + v[u][3]);
      bef = __reduce_add_sync(0xffffffffu, bef);
      float s = (f[u][0] + f[u][1]) + (f[u][2] + f[u][3]);
      if (finish)
#pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0 && e < n_experts) {
        total[e] = tot;
        before[e] = bef;
        colsum[e] = s;
      }
    }
  }
  // the pair's rank among its warp's (lower lane = lower pair id)
  int rank = 0;
  if (warp < warps) {
    const unsigned peers = __match_any_sync(0xffffffffu, e_mine);
    rank = __popc(peers & ((1u << lane) - 1u));
    if (e_mine >= 0 && rank == 0) mine[warp][e_mine] = uint16_t(__popc(peers));
  }
  __syncthreads();
  auto cap_of = [&](int e) { return sc.capacity > 0 && e < sc.n_capped ? sc.capacity : INT32_MAX; };
  if (warp == WARPS - 1) {
    // exclusive scan of the padded run lengths, 8 consecutive experts per lane
    constexpr int PER = MAX_EXPERTS / 32;
    int32_t pad[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane * PER + i;
      pad[i] = e < n_experts ? (min(total[e], cap_of(e)) + ALIGN_M - 1) / ALIGN_M * ALIGN_M : 0;
      sum += pad[i];
    }
    int32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    int32_t run = incl - sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane * PER + i;
      if (e <= n_experts) off[e] = run;
      run += pad[i];
    }
    if (lane == 31) off[MAX_EXPERTS] = run;
  } else if (warp == WARPS - 2 && finish) {
    FinishArgs fin = sc.fin;
    fin.colsum = block_colsum != nullptr ? colsum : nullptr;
    finish_forward<FINISH_SHARED>(fin, total, sc.capacity);
  }
  if (e_mine >= 0) {
    rank += before[e_mine];
    for (int w = 0; w < warp; ++w) rank += mine[w][e_mine];
  }
  __syncthreads();
  const int32_t live = off[n_experts];
  if (live_pair) {
    const bool kept = rank < cap_of(e_mine);
    const int32_t dst = kept ? off[e_mine] + rank : -1;
    if (kept) sorted_ids[dst] = int32_t(pair);
    sc.inv_ids[pair] = dst;
  }
  if (blk == 0) {
    for (int e = tid; e < n_experts; e += FRONT_THREADS) sc.counts[e] = total[e];
    for (int e = tid; e <= n_experts; e += FRONT_THREADS) sc.pad_offsets[e] = off[e];
    if (tid == 0) *sc.n_post_pad = live;
  }
  if (sc.expert_ids != nullptr) {   // every block its slice
    const int per = int((sc.n_tiles_cap + n_blocks - 1) / n_blocks);
    for (int i = tid; i < per && int64_t(per) * blk + i < sc.n_tiles_cap; i += FRONT_THREADS)
      sc.expert_ids[int64_t(per) * blk + i] = tile_owner(off, n_experts, live, int64_t(per) * blk + i);
  }
}

template <int NS>
static int launch_front(const FrontArgs& a, int epl, unsigned blocks, int smem, cudaStream_t st) {
  auto kern = router_front_kernel<NS>;
  static PerDevice<int> ready;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return MOE_B200_ERR_CUDA;
  const int* ok = ready.get(dev, [&](int) {
    return int(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FRONT_MAX_SMEM) ==
               cudaSuccess);
  });
  if (ok == nullptr || !*ok) return MOE_B200_ERR_CUDA;
  return launch_pdl(kern, dim3(blocks), dim3(FRONT_THREADS), size_t(smem), st, a, epl) == cudaSuccess
             ? MOE_B200_OK
             : MOE_B200_ERR_CUDA;
}

bool router_front_covers(int64_t n_tokens, int32_t d_model, int32_t n_experts, int32_t n_shared,
                         int32_t top_k, const void* x, const void* router_w) {
  return n_tokens >= 1 && n_tokens <= FRONT_TOKENS * FRONT_MAX_BLOCKS && d_model >= 64 &&
         d_model % 16 == 0 && n_experts >= 4 && n_experts % 4 == 0 && n_experts <= 128 &&
         top_k >= 1 && top_k <= RF4_MAX_TOPK && top_k <= n_experts && n_shared >= 0 &&
         top_k + n_shared <= 32 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 &&
         (reinterpret_cast<uintptr_t>(router_w) & 7u) == 0 &&
         front_smem(d_model, n_experts).total <= FRONT_MAX_SMEM;
}

size_t router_front_scratch_bytes(int64_t n_tokens, int32_t n_experts, int32_t n_shared) {
  if (n_tokens > FRONT_TOKENS * FRONT_MAX_BLOCKS) return 0;
  const int64_t blocks = (n_tokens + FRONT_TOKENS - 1) / FRONT_TOKENS;
  return size_t(blocks) * size_t(2 * n_experts + n_shared) * 4;
}

int router_front(const FrontCall& c, cudaStream_t st) {
  if (!router_front_covers(c.n_tokens, c.d_model, c.n_experts, c.n_shared, c.top_k, c.x, c.router_w))
    return MOE_B200_ERR_UNSUPPORTED;
  if (!c.x || !c.router_w || !c.w_all || !c.idx_all || !c.sorted_ids || !c.scratch || !c.status ||
      !c.scatter.counts || !c.scatter.pad_offsets || !c.scatter.n_post_pad || !c.scatter.inv_ids)
    return MOE_B200_ERR_NULL;
  const int blocks = int((c.n_tokens + FRONT_TOKENS - 1) / FRONT_TOKENS);
  const int n_all = c.n_experts + c.n_shared, kS = c.top_k + c.n_shared;
  FrontArgs a{};
  a.x = static_cast<const __nv_bfloat16*>(c.x);
  a.w = static_cast<const __nv_bfloat16*>(c.router_w);
  a.bias = c.bias;
  a.route = RouteArgs{c.noise, static_cast<__nv_bfloat16*>(c.w_all), c.idx_all, c.n_experts, c.top_k,
                      c.n_shared, c.normalize, c.full_softmax};
  a.n_tokens = c.n_tokens;
  a.d_model = c.d_model;
  a.logits = static_cast<__nv_bfloat16*>(c.logits);
  a.w_padded = static_cast<__nv_bfloat16*>(c.w_padded);
  a.ld = c.ld;
  a.block_hist = static_cast<int32_t*>(c.scratch);
  a.block_colsum = c.full_softmax ? reinterpret_cast<float*>(a.block_hist + blocks * n_all) : nullptr;
  a.sorted_ids = c.sorted_ids;
  a.l_cap = c.scatter.n_tiles_cap * ALIGN_M;
  a.status = c.status;
  const int smem = front_smem(c.d_model, c.n_experts).total;
  const int epl = rf4_lane_experts(c.n_experts);
  const int rc = c.n_experts <= 32   ? launch_front<1>(a, epl, unsigned(blocks), smem, st)
                 : c.n_experts <= 64 ? launch_front<2>(a, epl, unsigned(blocks), smem, st)
                 : c.n_experts <= 96 ? launch_front<3>(a, epl, unsigned(blocks), smem, st)
                                     : launch_front<4>(a, epl, unsigned(blocks), smem, st);
  if (rc != MOE_B200_OK) return rc;
  const cudaError_t err = launch_pdl(
      router_front_scatter_kernel, dim3(unsigned(blocks)), dim3(FRONT_THREADS), 0, st,
      static_cast<const int64_t*>(c.idx_all), int32_t(c.n_tokens * kS), n_all, FRONT_TOKENS * kS,
      static_cast<const int32_t*>(a.block_hist), static_cast<const float*>(a.block_colsum), c.sorted_ids,
      c.scatter);
  return err == cudaSuccess ? MOE_B200_OK : MOE_B200_ERR_CUDA;
}

}  // namespace moe
