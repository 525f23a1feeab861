// A token's routing in two forms with the same results to the bit: on four lanes (router_fused.cu, many
// tokens) and on a warp (router_front.cu, where the chain of one token counts).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "pdl.cuh"
#include "routing.cuh"

namespace moe {

constexpr int RF4_MAX_TOPK = 8;
// Experts per lane of the four-lane form (0: too many).
inline int rf4_lane_experts(int n_experts) {
  return n_experts <= 32 ? 8 : n_experts <= 64 ? 16 : n_experts <= 80 ? 20 : n_experts <= 96 ? 24
         : n_experts <= 128 ? 32 : 0;
}

__device__ __forceinline__ float key_float(uint32_t k) {   // inverse of float_key
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// a <- the KT largest of two descending lists of KT (max of one against the other reversed), sorted
// again if asked: a bitonic merge, or the 12-comparator network for 6.
template <int KT, bool SORT>
__device__ __forceinline__ void merge_top(uint32_t (&a)[KT], const uint32_t (&b)[KT]) {
#pragma unroll
  for (int j = 0; j < KT; ++j) a[j] = max(a[j], b[KT - 1 - j]);
  auto order = [&](int x, int y) {
    const uint32_t hi = max(a[x], a[y]), lo = min(a[x], a[y]);
    a[x] = hi;
    a[y] = lo;
  };
  if constexpr (SORT && KT == 6) {
    order(0, 5), order(1, 3), order(2, 4);
    order(1, 2), order(3, 4);
    order(0, 3), order(2, 5);
    order(0, 1), order(2, 3), order(4, 5);
    order(1, 2), order(3, 4);
  } else if constexpr (SORT) {
#pragma unroll
    for (int d = KT / 2; d > 0; d >>= 1)
#pragma unroll
      for (int j = 0; j < KT; ++j)
        if ((j & d) == 0) order(j, j + d);
  }
}

struct RouteArgs {
  const float* noise;        // [T, E] or null
  __nv_bfloat16* w_all;      // [T, k + S]
  int64_t* idx_all;          // [T, k + S]
  int32_t n_experts, top_k, n_shared, normalize, full_softmax;
};

// Lane q = lane & 3 of the token's group, with experts [e0, e0 + EPL), e0 = q * EPL; load(e) gives the
// logits of experts e..e+3 as 8 bytes. A lane whose token does not exist (!valid) works on token tc and
// writes nothing. list: the group's KT + 1 entries of shared memory; hist (may be null): counts per expert;
// csum: this lane's share of the column sums of the probabilities (COLSUM only).
template <int EPL, int KT, bool COLSUM, typename Load>
__device__ __forceinline__ void route_token(const RouteArgs& a, Load load, int64_t t, int64_t tc, bool valid,
                                            const float (&b)[EPL], float (&csum)[COLSUM ? EPL : 1],
                                            uint2* list, int32_t* hist) {
  const int lane = threadIdx.x & 31, q = lane & 3, e0 = q * EPL;
  const int kS = a.top_k + a.n_shared;
  const bool need_full = a.full_softmax || !a.normalize;
  uint32_t key[EPL];   // first the values (as float bits), then the order-preserving keys
  float mx = -CUDART_INF_F;
  {
    uint2 r[EPL / 4];
#pragma unroll
    for (int c = 0; c < EPL / 4; ++c)
      r[c] = e0 + 4 * c < a.n_experts ? load(e0 + 4 * c) : make_uint2(0u, 0u);
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const uint32_t w = (i & 2) ? r[i / 4].y : r[i / 4].x;
      const float f = __uint_as_float((i & 1) ? w & 0xffff0000u : w << 16);
      float v = e0 + i < a.n_experts ? f + b[i] : -CUDART_INF_F;
      if (a.noise != nullptr && e0 + i < a.n_experts)   // exploration noise, one value per (token, expert)
        v += ld_prev(a.noise + tc * a.n_experts + e0 + i);
      key[i] = __float_as_uint(v);
      mx = fmaxf(mx, v);
    }
  }
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));

  float denom = 0.f;
  if (need_full) {
    float ex[EPL];
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      ex[i] = (e0 + i < a.n_experts) ? expf(__uint_as_float(key[i]) - mx) : 0.f;
      denom += ex[i];
    }
    denom += __shfl_xor_sync(0xffffffffu, denom, 1);
    denom += __shfl_xor_sync(0xffffffffu, denom, 2);
    if constexpr (COLSUM) {
      const float inv = valid ? 1.f / denom : 0.f;
#pragma unroll
      for (int i = 0; i < EPL; ++i) csum[i] += ex[i] * inv;
    }
  }
  uint32_t top[KT];   // this lane's largest keys, descending
#pragma unroll
  for (int j = 0; j < KT; ++j) top[j] = 0u;
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    // (no key of a value is 0: that is what experts past the end get)
    const uint32_t x = e0 + i < a.n_experts ? float_key(__uint_as_float(key[i])) : 0u;
    key[i] = x;
#pragma unroll
    for (int j = KT - 1; j > 0; --j)
      if (j <= i) top[j] = max(top[j], min(top[j - 1], x));
    top[0] = max(top[0], x);
  }
  {
    uint32_t other[KT];
#pragma unroll
    for (int j = 0; j < KT; ++j) other[j] = __shfl_xor_sync(0xffffffffu, top[j], 1);
    merge_top<KT, true>(top, other);
#pragma unroll
    for (int j = 0; j < KT; ++j) other[j] = __shfl_xor_sync(0xffffffffu, top[j], 2);
    merge_top<KT, true>(top, other);
  }
  uint32_t last = 0xFFFFFFFFu;   // the smallest key that is in
#pragma unroll
  for (int j = 0; j < KT; ++j) last = min(last, j < a.top_k ? top[j] : 0xFFFFFFFFu);

  uint32_t in = 0u;   // this lane's experts that are in
#pragma unroll
  for (int i = 0; i < EPL; ++i)
    if (key[i] >= last) in |= 1u << i;
  int n = __popc(in);
  int total = n + __shfl_xor_sync(0xffffffffu, n, 1);
  total += __shfl_xor_sync(0xffffffffu, total, 2);
  if (__any_sync(0xffffffffu, total > a.top_k)) {
    // more ties for the last place than places: the highest experts among them are out
    uint32_t tie = 0u;
#pragma unroll
    for (int i = 0; i < EPL; ++i)
      if (key[i] == last) tie |= 1u << i;
    const int nt = __popc(tie);
    int over = total - a.top_k;
#pragma unroll
    for (int k = 3; k > 0; --k) {   // what the lanes above take
      const int up = __shfl_sync(0xffffffffu, nt, (lane & ~3) + k);
      if (k > q) over -= up;
    }
    for (over = min(over, nt); over > 0; --over) {
      const uint32_t bit = 0x80000000u >> __clz(tie);
      tie ^= bit;
      in ^= bit;
    }
    n = __popc(in);
  }
  int pos = n;
  {
    const int u1 = __shfl_up_sync(0xffffffffu, pos, 1);
    if (q >= 1) pos += u1;
    const int u2 = __shfl_up_sync(0xffffffffu, pos, 2);
    if (q >= 2) pos += u2;
    pos -= n;
  }
  __syncwarp();   // the previous token's list has been read
#pragma unroll
  for (int i = 0; i < EPL; ++i)
    if (in >> i & 1u) list[pos++] = make_uint2(key[i], uint32_t(e0 + i));
  __syncwarp();

  // lane q ranks entries q and q + 4: by value descending, then by index
  uint2 cand[KT];
#pragma unroll
  for (int j = 0; j < KT; ++j) cand[j] = j < a.top_k ? list[j] : make_uint2(0u, 0u);
  float p[2], s = 0.f;
  int rank[2], ei[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int me = q + 4 * h;
    const bool mine = me < a.top_k;
    const uint2 c = mine ? list[me] : make_uint2(0u, 0u);
    const float val = key_float(c.x);
    p[h] = !mine ? 0.f : need_full ? expf(val - mx) / denom : expf(val - mx);
    s += p[h];
    ei[h] = int(c.y);
    rank[h] = 0;
#pragma unroll
    for (int j = 0; j < KT; ++j)
      if (cand[j].x > c.x || (cand[j].x == c.x && j < me)) ++rank[h];
  }
  if (!need_full || (a.normalize && a.top_k > 1 && a.full_softmax)) {
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    p[0] = p[0] / s;
    p[1] = p[1] / s;
  }
  if (valid) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (q + 4 * h < a.top_k) {
        a.w_all[t * kS + rank[h]] = __float2bfloat16(p[h]);
        a.idx_all[t * kS + rank[h]] = ei[h];
        if (hist != nullptr) atomicAdd(&hist[ei[h]], 1);
      }
    for (int jj = a.top_k + q; jj < kS; jj += 4) {   // the shared experts: every token, weight 1
      a.w_all[t * kS + jj] = __float2bfloat16(1.f);
      a.idx_all[t * kS + jj] = a.n_experts + (jj - a.top_k);
    }
  }
}

// The same on a warp, for few tokens. What bounds that is not instructions but fetching them: straight-line
// code that runs once costs some ten cycles an instruction (the form above 8.7 us for 16 tokens on two
// warps, 10 with column sums), so the loops here stay rolled and short. Every sum runs in the order of the
// form above, whose lanes hold the experts in four parts of `epl`.
//   lg: the token's logits in shared memory; ex: room for E floats, left as the token's probabilities where
//   column sums are wanted; tmp: 8 floats. NS = ceil(E / 32).
template <int NS>
__device__ __forceinline__ void route_warp(const RouteArgs& a, const __nv_bfloat16* lg, const float* bias,
                                           int64_t t, int epl, float* ex, float* tmp, int32_t* hist) {
  const int lane = threadIdx.x & 31, E = a.n_experts, kS = a.top_k + a.n_shared;
  const bool need_full = a.full_softmax || !a.normalize;
  float v[NS];
  uint32_t key[NS];
  float mx = -CUDART_INF_F;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const int e = i * 32 + lane;
    v[i] = -CUDART_INF_F;
    key[i] = 0u;   // (no key of a value is 0)
    if (e < E) {
      v[i] = __bfloat162float(lg[e]) + (bias != nullptr ? ld_prev(bias + e) : 0.f);
      if (a.noise != nullptr) v[i] += ld_prev(a.noise + t * E + e);
      key[i] = float_key(v[i]);
    }
    mx = fmaxf(mx, v[i]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  uint32_t my_key = 0u;
  int my_idx = 0x7fffffff;
#pragma unroll 1
  for (int j = 0; j < a.top_k; ++j) {   // the j-th choice goes to lane j
    uint32_t best = key[0];
#pragma unroll
    for (int i = 1; i < NS; ++i) best = max(best, key[i]);
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    uint32_t cand = 0xFFFFFFFFu;
#pragma unroll
    for (int i = NS - 1; i >= 0; --i)
      if (key[i] == top) cand = uint32_t(i * 32 + lane);
    const int win = int(__reduce_min_sync(0xffffffffu, cand));
#pragma unroll
    for (int i = 0; i < NS; ++i)
      if (i * 32 + lane == win) key[i] = 0u;
    if (lane == j) {
      my_key = top;
      my_idx = win;
    }
  }
  float denom = 0.f;
  if (need_full) {
#pragma unroll
    for (int i = 0; i < NS; ++i)
      if (i * 32 + lane < E) ex[i * 32 + lane] = expf(v[i] - mx);
    __syncwarp();
    if (lane < 4) {   // four parts, each in order
      const int lo = lane * epl, hi = min(lo + epl, E);
#pragma unroll 4
      for (int e = lo; e < hi; ++e) denom += ex[e];
    }
    denom += __shfl_xor_sync(0xffffffffu, denom, 1);
    denom += __shfl_xor_sync(0xffffffffu, denom, 2);
    denom = __shfl_sync(0xffffffffu, denom, 0);
    const float inv = 1.f / denom;
#pragma unroll
    for (int i = 0; i < NS; ++i)
      if (i * 32 + lane < E) ex[i * 32 + lane] *= inv;
  }
  const bool mine = lane < a.top_k;
  float w = mine ? expf(key_float(my_key) - mx) : 0.f;
  if (need_full) w /= denom;
  if (!need_full || (a.normalize && a.top_k > 1 && a.full_softmax)) {
    // the choices in the order of their experts: entries 0..7, lane q of the form above has q and q + 4
    int pos = 0;
#pragma unroll 1
    for (int j = 0; j < a.top_k; ++j) pos += __shfl_sync(0xffffffffu, my_idx, j) < my_idx ? 1 : 0;
    if (lane < RF4_MAX_TOPK) tmp[lane] = 0.f;
    __syncwarp();
    if (mine) tmp[pos] = w;
    __syncwarp();
    float s = lane < 4 ? tmp[lane] + tmp[lane + 4] : 0.f;
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    w /= __shfl_sync(0xffffffffu, s, 0);
  }
  if (lane < kS) {
    a.w_all[t * kS + lane] = __float2bfloat16(mine ? w : 1.f);   // the shared experts: weight 1
    a.idx_all[t * kS + lane] = mine ? my_idx : E + (lane - a.top_k);
    if (mine) atomicAdd(&hist[my_idx], 1);
  }
}

}  // namespace moe
