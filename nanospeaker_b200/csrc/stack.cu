// A stack of MoE blocks on a small batch (decode: one token per sequence) as ONE persistent kernel:
// x <- x + block_l(x) for every layer, two grid-wide hand-overs per layer and nothing else between
// the layers.
//
// Layer by layer (five launches each) the stack took 38 us per layer at 1 token and 45 us at 64,
// against 5.3 us for reading the layer's 34.5 MB of weights: a chain of launch latencies, each
// launch holding a handful of rows in 128-row tiles. Here:
//   token phase   CTA t mod G owns token t: it sums the token's per-pair partial rows of the previous
//                 layer in a fixed order, adds the residual, rounds to bf16, forms the router logits
//                 against the row it has just made, and selects the experts.
//   expert phase  a work item is (expert, 32 of its 128 hidden units): 108 KB of weights at d_model
//                 576, so that the 312 items of 78 experts spread over 148 SMs. It takes the rows of
//                 the tokens that chose the expert, computes its hidden units (up/gate + GLU) and its
//                 share of the down product, and leaves fp32 partial rows [pair][slice].
// What it is bound by is the chain of latencies through the two phases, not the weights: which items
// a CTA owns depends on nothing but the shape, so the weights of the coming items (the next layer's
// included) stream into a shared-memory ring by TMA while the phases run; only the rows travel on
// the critical path. Rows per item are few (5 at 64 tokens), so the products are mma.sync m16n8k16
// with the weights as the 16-row operand: tcgen05 tiles would hold 5 rows in 128.
// Everything is summed in a fixed order: results are bit-reproducible.
//
// The grid is launched cooperatively (its CTAs wait on one another); every wait is bounded.
//
// Nearly every instruction runs once or twice per layer, so the code is as much on the critical path as
// the data: straight-line code that misses the small instruction caches costs some 20 cycles an
// instruction. Loops are kept rolled, rare variants out of line, and the weight loads are a few
// instructions of one warp (176 KB of unrolled code: 27 us a layer at 64 tokens).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <cstring>

#include "../../include/moe_b200.h"
#include "act.cuh"
#include "agree.cuh"
#include "pdl.cuh"
#include "ptx.cuh"
#include "routing.cuh"
#include "stack_shape.cuh"
#include "tma_map.cuh"

namespace moe {

static_assert(ST_MAX_GROUPS == MAX_EXPERTS, "the routing kernels take as many");

struct alignas(64) StackLayer {
  CUtensorMap in, out, sh_in, sh_out;
  const __nv_bfloat16* router_w;           // [D, E]
  const float* bias;                       // [E] or null
};

struct StackArgs {
  const StackLayer* layers;
  int32_t n_layers, T, D, E, S, k, normalize, act;
  int32_t n_stages;                        // of the ring
  int32_t router_extra;                    // bytes of shared memory for router weight chunks alone
  int32_t out_boxes;                       // TMA boxes per down stage: 1, or 2 when d_model % 64 != 0
  int32_t kshift;                          // idx rows hold 1 << kshift entries: 8 or 16
  int32_t sh_tokens, sh_blocks;            // a shared expert's tokens are cut into blocks
  int32_t n_items;                         // per layer: S * slices * sh_blocks, then E * slices
  const __nv_bfloat16* x;
  __nv_bfloat16* out;
  __nv_bfloat16* xbuf;                     // [T, D] the residual stream
  float* partial;                          // [T * (k + S)][slices][D]
  uint16_t* idx;                           // [T][1 << kshift] chosen experts, 0xffff beyond k
  uint32_t* ctr;                           // [2] arrivals of the token / expert phase (start at 0)
  int32_t* status;
};

struct StackItem {
  int expert;        // < E routed, else shared
  int slice, t0, n;  // shared: its token block; routed: n = -1
};
__host__ __device__ __forceinline__ int stack_position(int r, int cta, int grid) {
  return r * grid + ((r & 1) ? grid - 1 - cta : cta);   // up and down: the last, partial round's extra
}                                                       // items go to CTAs without a shared one
__device__ __forceinline__ StackItem stack_item(const StackArgs& p, int pos) {
  StackItem it;
  const int n_sh = p.S * ST_SLICES * p.sh_blocks;
  if (pos < n_sh) {
    const int blk = pos / (p.S * ST_SLICES), rest = pos - blk * p.S * ST_SLICES;
    it.expert = p.E + rest / ST_SLICES;
    it.slice = rest % ST_SLICES;
    it.t0 = blk * p.sh_tokens;
    it.n = min(p.sh_tokens, p.T - it.t0);
  } else {
    it.expert = (pos - n_sh) / ST_SLICES;
    it.slice = (pos - n_sh) % ST_SLICES;
    it.t0 = 0;
    it.n = -1;
  }
  return it;
}

// ------------------------------------------------------------------------------ small PTX
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ct_sync() {   // the compute warps
  asm volatile("bar.sync 1, %0;" ::"n"(ST_CT) : "memory");
}
__device__ __forceinline__ void arrive_gpu(uint32_t* ctr) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
}
__device__ __forceinline__ uint32_t load_gpu(const uint32_t* ctr) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ldcg4(const float* p) {
  return __ldcg(reinterpret_cast<const float4*>(p));
}
__device__ __noinline__ float stack_other_act(int act, float g) {
  switch (act) {
    case ACT_GELU: return act_f<ACT_GELU>(g);
    case ACT_RELU: return act_f<ACT_RELU>(g);
    case ACT_SIGMOID: return act_f<ACT_SIGMOID>(g);
    default: return act_f<ACT_TANH>(g);
  }
}
__device__ __forceinline__ float stack_act(int act, float g) {
  return act == ACT_SILU ? act_f<ACT_SILU>(g) : stack_other_act(act, g);
}
// A value that the compiler cannot reason about: keeps it from cloning loops for their special cases.
__device__ __forceinline__ int opaque(int v) {
  asm volatile("" : "+r"(v));
  return v;
}

// One warp: the k largest of lg[0, E) (value descending, ties to the lowest index; keys[e] is
// float_key of lg[e], at least 1) and their softmax weights, rounded to bf16. NS = ceil(E / 32) values
// per lane. Lane j returns the j-th choice.
template <int NS>
__device__ __forceinline__ void stack_select(const float* lg, const uint32_t* keys, int E, int k,
                                             int normalize, int lane, int* idx, float* weight) {
  uint32_t key[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) key[i] = i * 32 + lane < E ? keys[i * 32 + lane] : 0u;
  int sel = 0;
#pragma unroll 1
  for (int j = 0; j < k; ++j) {
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
    if (lane == j) sel = win;
  }
  const bool active = lane < k;   // (k <= 16)
  const float val = lg[sel];
  const float top = __shfl_sync(0xffffffffu, val, 0);
  const float ex = active ? expf(val - top) : 0.f;
  float s = ex;
  if (normalize) {
#pragma unroll
    for (int o = 8; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  } else {
    s = 0.f;
#pragma unroll 1
    for (int e = lane; e < E; e += 32) s += expf(lg[e] - top);
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  *idx = active ? sel : 0xffff;
  *weight = active ? __bfloat162float(__float2bfloat16(ex / s)) : 1.f;   // past k: the shared experts
}

template <int SELECT>   // values per lane in the expert selection: at most 32 * SELECT experts
__global__ void __launch_bounds__(ST_THREADS, 1) stack_kernel(const StackArgs p) {
  extern __shared__ uint8_t smem_raw[];
  // (aligned by an offset, not through an integer: the accesses stay shared-memory ones)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const StackSmem L = stack_smem(p.T, p.D, p.n_stages, p.router_extra);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bars);   // [ST_PARTS] up / down weights of an item
  uint64_t* empty = full + ST_PARTS;                             // [ST_PARTS] their stages are free again
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.misc);
  volatile int* go_on = abort_flag + 1;   // written by compute thread 0 alone
  int* cnt = reinterpret_cast<int*>(smem + L.misc + 16);
  StackItem* items = reinterpret_cast<StackItem*>(smem + L.misc + 16 + ST_MAX_ITEMS * 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = int(gridDim.x), cta = int(blockIdx.x);
  const int D = p.D, dpad = (D + 63) / 64 * 64;
  const int n_in = dpad / 64, n_out = (n_in + 1) / 2;   // ring stages of one item
  const int NS = p.n_stages;
  const int kS = p.k + p.S;
  // this CTA's items (all but the last round are full)
  const int rounds = (p.n_items + G - 1) / G;
  const int n_mine = rounds - (stack_position(rounds - 1, cta, G) < p.n_items ? 0 : 1);

  if (tid == 0) {
    for (int s = 0; s < 2 * ST_PARTS; ++s) mbar_init(full + s, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (tid < n_mine) items[tid] = stack_item(p, stack_position(tid, cta, G));
  __syncthreads();
  pdl_wait();   // the counters, x and the weights may come from the kernels before this one

  if (warp == ST_WARPS) {
    // ------------------------------------------------------------------ weights by TMA
    if (elect_one() && n_mine > 0) {
      int slot = 0, part = 0;            // of the ring; of the loads
      int ahead = NS, old_part = 0;      // stages until the next part's have to be free; that part
      bool ok = true;
#pragma unroll 1
      for (int l = 0; l < p.n_layers && ok; ++l) {
#pragma unroll 1
        for (int r = 0; r < 2 * n_mine && ok; ++r, ++part) {   // up, down of every item
          const StackItem item = items[r >> 1];
          const bool shared = item.expert >= p.E, down = r & 1;
          // (a layer's maps lie in the order in, out, sh_in, sh_out)
          const CUtensorMap* map = &p.layers[l].in + (shared ? 2 : 0) + (down ? 1 : 0);
          const int g = shared ? item.expert - p.E : item.expert, u = item.slice * ST_SLICE;
          const int n = down ? n_out : n_in;
          uint64_t* bar = full + part % ST_PARTS;
#pragma unroll 1
          for (int c = 0; c < n && ok; ++c) {
            if (ahead == 0) {   // this stage was part old_part's
              ok = mbar_wait(empty + old_part % ST_PARTS, (old_part / ST_PARTS) & 1, p.status) &&
                   *abort_flag == 0;
              if (!ok) break;
              ahead = old_part & 1 ? n_out : n_in;
              ++old_part;
            }
            --ahead;
            if (c == 0) mbar_expect_tx(bar, n * ST_STAGE);
            uint8_t* dst = smem + slot * ST_STAGE;
            if (!down) {
              tma_load_4d(dst, map, bar, u, c * 64, 0, g);
            } else if (p.out_boxes == 1) {
              tma_load_4d(dst, map, bar, 0, u, 2 * c, g);
            } else {
              tma_load_3d(dst, map, bar, c * 128, u, g);
              tma_load_3d(dst + ST_HALF, map, bar, c * 128 + 64, u, g);
            }
            if (++slot == NS) slot = 0;
          }
        }
      }
      if (!ok) {   // given up: let what is in flight land before the CTA may leave
        *abort_flag = 1;
        atomicExch(p.status, ST_WAIT_TIMEOUT);
        __nanosleep(1000000);
      }
    }
    return;
  }

  // ---------------------------------------------------------------------- compute warps
  const uint32_t ring_u = smem_u32(smem), xs_u = smem_u32(smem + L.xs);
  const uint32_t xs_ld = dpad * 2 + 16;
  float* acc_s = reinterpret_cast<float*>(smem + L.acc);
  float* red_s = reinterpret_cast<float*>(smem + L.acc + ST_ACC_BYTES - ST_RED_BYTES);
  __nv_bfloat16* hid_s = reinterpret_cast<__nv_bfloat16*>(smem + L.hid);
  uint16_t* list = reinterpret_cast<uint16_t*>(smem + L.list);   // [item][tokens | pairs][T]
  float* xrow = reinterpret_cast<float*>(smem + L.xrow);
  __nv_bfloat16* res = reinterpret_cast<__nv_bfloat16*>(smem + L.res);
  float* tokw = reinterpret_cast<float*>(smem + L.tokw);
  float* lg = reinterpret_cast<float*>(smem + L.lg);
  uint32_t* keys = reinterpret_cast<uint32_t*>(smem + L.lg) + MAX_EXPERTS;
  const int token_ctas = min(p.T, G);
  const bool has_token = cta < p.T;
  const int kpad = 1 << p.kshift;

  // One thread looks at the counter and at the abort flag (which the TMA warp, outside the compute
  // warps' barrier, sets at any time), the CTA follows. False: given up.
  auto grid_wait = [&](const uint32_t* ctr, uint32_t target) {
    const bool go = agree(tid == 0, go_on, [&] {
      uint32_t n = 0;
#pragma unroll 1
      while (load_gpu(ctr) < target) {
        if (++n > (1u << 22) || ((n & 1023u) == 0 && *reinterpret_cast<volatile int32_t*>(p.status))) {
          atomicExch(p.status, ST_WAIT_TIMEOUT);
          *abort_flag = 1;
          break;
        }
      }
      return *abort_flag == 0;
    }, ct_sync);
    if (!go && tid == 0) __nanosleep(1000000);   // let the loads in flight land before the CTA leaves
    return go;
  };
  int ring_s = 0, part = 0;   // the ring as the consumers see it: the current item's first stage, its part
  auto part_wait = [&](int q) {
    if (!mbar_wait(full + q % ST_PARTS, (q / ST_PARTS) & 1, p.status)) {
      atomicExch(p.status, ST_WAIT_TIMEOUT);
      *abort_flag = 1;
    }
  };

  // router weight: a thread owns four columns (4 * (tid % P)) of every Q-th row
  const int P = p.E / 4, Q = ST_CT / P;
  const int rp = tid % P, rq = tid / P;
  const int router_rows = rq < Q ? (D - rq + Q - 1) / Q : 0;
  const int router_room = (p.router_extra + L.acc - L.xs + ST_ACC_BYTES - ST_RED_BYTES) / (ST_CT * 8);
  uint8_t* router_s = smem + L.xs - p.router_extra;
  const int cg = D / 4, groups = ST_CT / cg;   // token phase: 16-byte column groups, sets of pairs
  const __nv_bfloat16* rw = p.layers[0].router_w;   // (the next layer's are fetched a layer ahead)
  const float* bias = p.layers[0].bias;

#pragma unroll 1
  for (int l = 0;; l = opaque(l + 1)) {   // (leaves in the token phase behind the last layer)
    const bool last = opaque(l) == p.n_layers;
    // ------------------------------------------------------------------ token phase
    if (has_token) {
      uint2 wr[ST_ROUTER_PRE];   // (on its way while this CTA waits for the others' partial rows)
      const uint2* rsrc = reinterpret_cast<const uint2*>(rw + rq * p.E + 4 * rp);
      const int rstep = Q * P, rn = last ? 0 : router_rows;   // (in chunks of four columns)
#pragma unroll
      for (int i = 0; i < ST_ROUTER_PRE; ++i)
        wr[i] = i < rn ? ld_prev(rsrc + i * rstep) : make_uint2(0u, 0u);
#pragma unroll 1
      for (int i = ST_ROUTER_PRE; i < min(rn, ST_ROUTER_PRE + router_room); ++i)
        cp_async_8(smem_u32(router_s) + ((i - ST_ROUTER_PRE) * ST_CT + tid) * 8, rsrc + i * rstep);
      cp_async_commit();
      if (opaque(l) > 0 && !grid_wait(p.ctr + 1, uint32_t(l) * G)) return;
#pragma unroll 1
      for (int t = cta, slot = 0; t < p.T; t += G, ++slot) {
        const bool first = opaque(l) == 0, last = opaque(l) == p.n_layers;
        __nv_bfloat16* my_res = res + slot * D;
        float* my_w = tokw + slot * 16;
        // the row: residual + the pairs' rows in order, each the sum of its slices' partial rows; four
        // columns per thread, the pairs cut into `groups` interleaved sets
        if (!first && tid < groups * cg) {
          const int g = tid / cg, c = tid - g * cg;
          const float* base = p.partial + int64_t(t) * kS * ST_SLICES * D + 4 * c;
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
          for (int j0 = g; j0 < kS; j0 += 3 * groups) {
            float4 v[3][ST_SLICES];
#pragma unroll
            for (int u = 0; u < 3; ++u)
#pragma unroll
              for (int q = 0; q < ST_SLICES; ++q)
                v[u][q] = ldcg4(base + (min(j0 + u * groups, kS - 1) * ST_SLICES + q) * D);
#pragma unroll
            for (int u = 0; u < 3; ++u) {
              const float w = j0 + u * groups < kS ? my_w[j0 + u * groups] : 0.f;
              a.x += w * ((v[u][0].x + v[u][1].x) + (v[u][2].x + v[u][3].x));
              a.y += w * ((v[u][0].y + v[u][1].y) + (v[u][2].y + v[u][3].y));
              a.z += w * ((v[u][0].z + v[u][1].z) + (v[u][2].z + v[u][3].z));
              a.w += w * ((v[u][0].w + v[u][1].w) + (v[u][2].w + v[u][3].w));
            }
          }
          *reinterpret_cast<float4*>(red_s + g * D + 4 * c) = a;
        }
        uint2 wl[ST_ROUTER_LATE];
        const int i_late = ST_ROUTER_PRE + router_room;
#pragma unroll
        for (int u = 0; u < ST_ROUTER_LATE; ++u)
          wl[u] = i_late + u < rn ? ld_prev(rsrc + (i_late + u) * rstep) : make_uint2(0u, 0u);
        ct_sync();
#pragma unroll 1
        for (int d = 2 * tid; d < dpad; d += 2 * ST_CT) {
          float v0 = 0.f, v1 = 0.f;
          if (d < D) {
            __nv_bfloat162 h;
            if (!first) {
              const float2 f = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(my_res + d));
              v0 = f.x;
              v1 = f.y;
#pragma unroll 1
              for (int g = 0; g < groups; ++g) {
                const float2 r = *reinterpret_cast<const float2*>(red_s + g * D + d);
                v0 += r.x;
                v1 += r.y;
              }
              h = __floats2bfloat162_rn(v0, v1);
            } else {
              h = *reinterpret_cast<const __nv_bfloat162*>(p.x + int64_t(t) * D + d);
            }
            *reinterpret_cast<__nv_bfloat162*>(my_res + d) = h;
            *reinterpret_cast<__nv_bfloat162*>((last ? p.out : p.xbuf) + int64_t(t) * D + d) = h;
            const float2 f = __bfloat1622float2(h);
            v0 = f.x;
            v1 = f.y;
          }
          *reinterpret_cast<float2*>(xrow + d) = make_float2(v0, v1);
        }
        ct_sync();
        if (last) continue;
        if (rq < Q) {
          float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
          auto add = [&](uint2 w, float x) {
            a0 += x * __uint_as_float(w.x << 16);
            a1 += x * __uint_as_float(w.x & 0xffff0000u);
            a2 += x * __uint_as_float(w.y << 16);
            a3 += x * __uint_as_float(w.y & 0xffff0000u);
          };
#pragma unroll
          for (int i = 0; i < ST_ROUTER_PRE; ++i) add(wr[i], xrow[min(rq + i * Q, D - 1)]);
          cp_async_wait<0>();   // (a thread reads back what it copied itself)
          const uint2* ws = reinterpret_cast<const uint2*>(router_s) + tid;
          int i = ST_ROUTER_PRE;
#pragma unroll 2
          for (; i < min(rn, ST_ROUTER_PRE + router_room); ++i)
            add(ws[(i - ST_ROUTER_PRE) * ST_CT], xrow[rq + i * Q]);
#pragma unroll 1
          for (; i < rn; i += ST_ROUTER_LATE) {
#pragma unroll
            for (int u = 0; u < ST_ROUTER_LATE; ++u) add(wl[u], xrow[min(rq + (i + u) * Q, D - 1)]);
#pragma unroll
            for (int u = 0; u < ST_ROUTER_LATE; ++u)
              wl[u] = i + ST_ROUTER_LATE + u < rn ? ld_prev(rsrc + (i + ST_ROUTER_LATE + u) * rstep)
                                                  : make_uint2(0u, 0u);
          }
          *reinterpret_cast<float4*>(red_s + rq * p.E + 4 * rp) = make_float4(a0, a1, a2, a3);
        }
        const float b = bias != nullptr && tid < p.E ? ld_prev(bias + tid) : 0.f;
        ct_sync();
        if (tid < p.E) {   // (at most 256 experts: one thread each)
          float s = 0.f;
#pragma unroll 4
          for (int q = 0; q < Q; ++q) s += red_s[q * p.E + tid];
          s = __bfloat162float(__float2bfloat16(s)) + b;
          lg[tid] = s;
          keys[tid] = max(float_key(s), 1u);
        }
        ct_sync();
        if (warp == 0) {
          int sel;
          float w;
          stack_select<SELECT>(lg, keys, p.E, p.k, p.normalize, lane, &sel, &w);
          if (lane < kpad) p.idx[t * kpad + lane] = uint16_t(sel);
          if (lane < kS) my_w[lane] = w;
        }
        ct_sync();
      }
      if (last) return;
      if (tid == 0) arrive_gpu(p.ctr);   // (release: what the barrier above has collected)
    } else if (last) {
      return;
    }
    if (l + 1 < p.n_layers) {
      rw = p.layers[l + 1].router_w;
      bias = p.layers[l + 1].bias;
    }
    if (!grid_wait(p.ctr, uint32_t(l + 1) * token_ctas)) return;

    // ------------------------------------------------------------------ expert phase
    // Warp r lists the tokens of the CTA's r-th item (in any fixed order: a token's results do not
    // depend on its place in the list).
    if (warp < n_mine) {
      const StackItem item = items[warp];
      uint16_t *tok = list + 2 * warp * p.T, *pair = tok + p.T;
      int n = 0;
      if (item.n >= 0) {
#pragma unroll 1
        for (int i = lane; i < item.n; i += 32) {
          tok[i] = uint16_t(item.t0 + i);
          pair[i] = uint16_t((item.t0 + i) * kS + p.k + (item.expert - p.E));
        }
        n = item.n;
      } else {
        auto entries = [&](int b) {
          return b < p.T * kpad ? __ldcg(reinterpret_cast<const uint4*>(p.idx + b))
                                : make_uint4(~0u, ~0u, ~0u, ~0u);
        };
        uint4 next = entries(lane * 8);
#pragma unroll 1
        for (int b = lane * 8; b - lane * 8 < p.T * kpad; b += 256) {
          const uint4 v = next;
          next = entries(b + 256);
          // the place of the expert among the eight entries: a token chooses an expert once, and
          // eight entries are one token's (or half of one's)
          const uint32_t e2 = uint32_t(item.expert) * 0x10001u;
          const uint32_t h0 = __vcmpeq2(v.x, e2) & 0x00020001u, h1 = __vcmpeq2(v.y, e2) & 0x00080004u;
          const uint32_t h2 = __vcmpeq2(v.z, e2) & 0x00200010u, h3 = __vcmpeq2(v.w, e2) & 0x00800040u;
          const uint32_t h = h0 | h1 | h2 | h3, hits = (h | (h >> 16)) & 0xffu;
          const unsigned m = __ballot_sync(0xffffffffu, hits != 0);
          if (hits) {
            const int i = n + __popc(m & ((1u << lane) - 1u)), at = b + __ffs(hits) - 1;
            const int t = at >> p.kshift;
            tok[i] = uint16_t(t);
            pair[i] = uint16_t(t * kS + (at & (kpad - 1)));
          }
          n += __popc(m);
        }
      }
      if (lane == 0) cnt[warp] = n;
    }
    ct_sync();
    // The rows of the pass after (r, n0) -- the same item's next tokens, or the next item that has any --
    // are fetched as soon as this pass has read its own; a warp has one row.
    auto gather_next = [&](int r, int n0) {
      n0 += ST_PASS;
      if (r < 0 || n0 >= cnt[r]) {
        n0 = 0;
#pragma unroll 1
        do ++r;
        while (r < n_mine && cnt[r] == 0);
      }
      if (r < n_mine && warp < cnt[r] - n0) {
        const __nv_bfloat16* src = p.xbuf + int(list[2 * r * p.T + n0 + warp]) * D + lane * 8;
        uint32_t dst = xs_u + warp * xs_ld + lane * 16;
#pragma unroll 1
        for (int c = lane * 8; c < dpad; c += 256, src += 256, dst += 512)
          cp_async_16(dst, c < D ? src : p.xbuf, c < D ? 16u : 0u);
      }
      cp_async_commit();
    };
    gather_next(-1, 0);
    // The arrival does not wait for what only moves the ring on: a release stands in the memory pipe
    // behind the loads issued before it.
    int last_live = n_mine - 1;
#pragma unroll 1
    while (last_live >= 0 && cnt[last_live] == 0) --last_live;
    if (last_live < 0 && tid == 0) arrive_gpu(p.ctr + 1);
#pragma unroll 1
    for (int r = 0; r < n_mine; ++r) {
      const int n = cnt[r];
      // (an item that nobody chose only moves the ring on)
#pragma unroll 1
      for (int half = 0; half < 2; ++half, ++part) {   // up/gate, then down; each gives its stages back
        if (n == 0) {
          if (tid == 0) part_wait(part);
        } else if (half == 0) {
          // up/gate + GLU: 64 outputs (gate, up: two mma rows each) x 16 tokens; the four warps of an
          // mma row take a quarter of every 64-deep stage each
          const int mt = warp & 3, kp = warp >> 2;
#pragma unroll 1
          for (int n0 = 0; n0 < n; n0 += ST_PASS) {
            const int nn = min(ST_PASS, n - n0);
            cp_async_wait<0>();
            ct_sync();
            if (n0 == 0) part_wait(part);
            float acc[2][2][4] = {};   // [even / odd stages][column tile]
            const int a_k = kp * 16 + (lane & 7) + ((lane >> 4) & 1) * 8;
            const int a_c = (mt & 1) * 2 + ((lane >> 3) & 1);
            const uint32_t a0 = ring_u + (mt >> 1) * ST_HALF + a_k * 64 + ((a_c ^ ((a_k >> 1) & 3)) << 4);
            // (the second column tile's rows may be stale: their columns are not used)
            uint32_t b_addr = xs_u + (kp * 16 + ((lane >> 3) & 1) * 8) * 2 +
                              ((lane & 7) + ((lane >> 4) & 1) * 8) * xs_ld;
            uint32_t a_addr = a0 + ring_s * ST_STAGE;
            const uint32_t a_end = a0 + NS * ST_STAGE;
#pragma unroll 1
            for (int c = 0; c < n_in; c += 3, b_addr += 384) {
              uint32_t a[3][4], b[3][4];
#pragma unroll
              for (int u = 0; u < 3; ++u) {   // (behind the last stage: repeated, and not used)
                ldsm4_t(a_addr, a[u]);
                ldsm4(c + u < n_in ? b_addr + u * 128 : b_addr, b[u]);
                a_addr += ST_STAGE;
                if (a_addr == a_end) a_addr = a0;
              }
#pragma unroll
              for (int u = 0; u < 3; ++u)
                if (c + u < n_in) {
                  mma_bf16(acc[u & 1][0], a[u], b[u][0], b[u][1]);
                  mma_bf16(acc[u & 1][1], a[u], b[u][2], b[u][3]);
                }
            }
            float* dst = acc_s + (kp * ST_PASS + 2 * (lane & 3)) * ST_ACC_LD + mt * 16 + (lane >> 2);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              float* d = dst + 8 * q * ST_ACC_LD;
              d[0] = acc[0][q][0] + acc[1][q][0];
              d[ST_ACC_LD] = acc[0][q][1] + acc[1][q][1];
              d[8] = acc[0][q][2] + acc[1][q][2];
              d[ST_ACC_LD + 8] = acc[0][q][3] + acc[1][q][3];
            }
            ct_sync();
            gather_next(r, n0);
            if (warp < nn) {   // a warp: the 32 units of a token
              float g = 0.f, up = 0.f;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                g += acc_s[(q * ST_PASS + warp) * ST_ACC_LD + lane];
                up += acc_s[(q * ST_PASS + warp) * ST_ACC_LD + 32 + lane];
              }
              hid_s[(n0 + warp) * ST_HID_LD + lane] = __float2bfloat16(stack_act(p.act, g) * up);
            }
          }
        } else {
          // down: D outputs in rows of 16, 32 deep; a warp takes every 16th row
          part_wait(part);
          const uint16_t* pair = list + (2 * r + 1) * p.T;
          float* out0 = p.partial + items[r].slice * D + (lane >> 2);
          const int u0 = (lane & 7) + ((lane >> 4) & 1) * 8, c0 = (lane >> 3) & 1;
#pragma unroll 1
          for (int n0 = 0; n0 < n; n0 += ST_PASS) {
            uint32_t b[2][4];
            const uint32_t h_addr = smem_u32(hid_s) +
                                    (n0 + (lane & 7) + ((lane >> 4) & 1) * 8) * (ST_HID_LD * 2) +
                                    ((lane >> 3) & 1) * 16;
            ldsm4(h_addr, b[0]);
            ldsm4(h_addr + 32, b[1]);
            int dst[4];   // this thread's four tokens: where their rows begin, or -1
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int i = n0 + 8 * (q >> 1) + 2 * (lane & 3) + (q & 1);
              dst[q] = i < n ? int(pair[i]) * (ST_SLICES * D) : -1;
            }
#pragma unroll 1
            for (int m = warp; m < D / 16; m += ST_WARPS) {
              uint32_t a[2][4];
              int s = ring_s + (m >> 3);
#pragma unroll 1
              while (s >= NS) s -= NS;
              const uint32_t box = ring_u + s * ST_STAGE + ((m >> 2) & 1) * ST_HALF +
                                   u0 * 128 + ((((m & 3) * 2 + c0) ^ (u0 & 7)) << 4);
              ldsm4_t(box, a[0]);
              ldsm4_t(box + 16 * 128, a[1]);
              float acc[2][4] = {};
              mma_bf16(acc[0], a[0], b[0][0], b[0][1]);
              mma_bf16(acc[1], a[0], b[0][2], b[0][3]);
              mma_bf16(acc[0], a[1], b[1][0], b[1][1]);
              mma_bf16(acc[1], a[1], b[1][2], b[1][3]);
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (dst[q] >= 0) {
                  float* d = out0 + dst[q] + m * 16;
                  d[0] = acc[q >> 1][q & 1];
                  d[8] = acc[q >> 1][2 + (q & 1)];
                }
            }
          }
        }
        if (n > 0) ct_sync();
        if (tid == 0) mbar_arrive(empty + part % ST_PARTS);
        if (r == last_live && half == 1 && tid == 0) arrive_gpu(p.ctr + 1);
        const int freed = half == 0 ? n_in : n_out;
        ring_s = ring_s + freed < NS ? ring_s + freed : ring_s + freed - NS;
      }
    }
  }
}

// ---------------------------------------------------------------------------------- host
static StackDevice look_at(int device) {
  StackDevice d;
  int coop = 0;
  auto ready = [&](const void* kern) {   // its CTAs per SM, with all the shared memory it may ask for
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_MAX_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, ST_THREADS, ST_MAX_SMEM) != cudaSuccess)
      return 0;
    return n;
  };
  if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess)
    d.blocks_per_sm = std::min(ready(reinterpret_cast<const void*>(stack_kernel<3>)),
                               ready(reinterpret_cast<const void*>(stack_kernel<8>)));
  d.cooperative = coop != 0;
  cudaGetLastError();
  return d;
}
static const StackDevice& stack_device() {
  static const StackDevice none = {148, 1, true};   // without a device: the shape alone decides
  static PerDevice<StackDevice> devices;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return none;
  }
  const StackDevice* d = devices.get(dev, look_at);
  return d != nullptr ? *d : none;
}

__global__ void stack_reset_kernel(uint32_t* ctr) {
  pdl_wait();
  if (threadIdx.x < 2) ctr[threadIdx.x] = 0u;
}

struct StackScratch {
  uint32_t* ctr;
  __nv_bfloat16* xbuf;
  uint16_t* idx;
  float* partial;
  size_t total;
};
static StackScratch stack_scratch(void* base, int64_t T, int D, int S, int k) {
  size_t at = 0;
  auto take = [&](size_t bytes) {
    char* r = base ? static_cast<char*>(base) + at : nullptr;
    at += (bytes + 255) / 256 * 256;
    return r;
  };
  StackScratch s;
  s.ctr = reinterpret_cast<uint32_t*>(take(256));
  s.xbuf = reinterpret_cast<__nv_bfloat16*>(take(size_t(T) * D * 2));
  s.idx = reinterpret_cast<uint16_t*>(take(size_t(T) * (k <= 8 ? 8 : 16) * 2));
  s.partial = reinterpret_cast<float*>(take(size_t(T) * (k + S) * ST_SLICES * D * 4));
  s.total = at;
  return s;
}

}  // namespace moe

using namespace moe;

extern "C" {

int moe_b200_stack_supported(int64_t n_tokens, int32_t d_model, int32_t d_hidden,
                             int32_t n_experts, int32_t n_shared, int32_t top_k) {
  StackShape o;
  return stack_shape(stack_device(), n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, &o) ? 1 : 0;
}

size_t moe_b200_stack_plan_bytes(int32_t n_layers) {
  return n_layers < 1 ? 0 : size_t(n_layers) * sizeof(StackLayer);
}

size_t moe_b200_stack_scratch_bytes(int64_t n_tokens, int32_t d_model, int32_t n_shared,
                                    int32_t top_k) {
  if (n_tokens < 1 || d_model < 1 || n_shared < 0 || top_k < 1) return 0;
  return stack_scratch(nullptr, n_tokens, d_model, n_shared, top_k).total;
}

int moe_b200_stack_plan(void* host_plan, int32_t n_layers, int32_t layer, const void* router_w,
                        const float* logit_bias, const void* w_in, const void* w_out,
                        const void* w_sh_in, const void* w_sh_out, int32_t n_experts,
                        int32_t n_shared, int32_t d_model, int32_t d_hidden) {
  if (n_layers < 1 || layer < 0 || layer >= n_layers || n_experts < 1 || n_shared < 0 ||
      d_hidden != ST_H || d_model < 64 || d_model % 32 != 0)
    return MOE_B200_ERR_SHAPE;
  if (!host_plan || !router_w || !w_in || !w_out || (n_shared > 0 && (!w_sh_in || !w_sh_out)))
    return MOE_B200_ERR_NULL;
  const auto odd = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; };
  if (odd(router_w) || odd(w_in) || odd(w_out) || odd(w_sh_in) || odd(w_sh_out))
    return MOE_B200_ERR_ALIGN;
  StackLayer ly;
  std::memset(&ly, 0, sizeof(ly));
  const auto maps = [&](CUtensorMap* in, CUtensorMap* out, const void* wi, const void* wo, int g) {
    // W_in [g][gate | up][d][128] (strides in that order of the box): 32 columns of 64 rows of both
    const uint64_t di[4] = {uint64_t(d_hidden), uint64_t(d_model), 2, uint64_t(g)};
    const uint64_t si[3] = {uint64_t(4 * d_hidden), uint64_t(2 * d_hidden),
                            uint64_t(4 * d_hidden) * d_model};
    const uint32_t bi[4] = {ST_SLICE, 64, 2, 1};
    if (!make_map(in, wi, 4, di, si, bi, CU_TENSOR_MAP_SWIZZLE_64B)) return false;
    if (d_model % 64 == 0) {   // W_out [g][128][d / 64][64]: two column blocks of 32 rows
      const uint64_t dn[4] = {64, uint64_t(d_hidden), uint64_t(d_model / 64), uint64_t(g)};
      const uint64_t sn[3] = {uint64_t(2 * d_model), 128, uint64_t(2 * d_model) * d_hidden};
      const uint32_t bn[4] = {64, ST_SLICE, 2, 1};
      return make_map(out, wo, 4, dn, sn, bn);
    }
    const uint64_t dn[3] = {uint64_t(d_model), uint64_t(d_hidden), uint64_t(g)};
    const uint64_t sn[2] = {uint64_t(2 * d_model), uint64_t(2 * d_model) * d_hidden};
    const uint32_t bn[3] = {64, ST_SLICE, 1};
    return make_map(out, wo, 3, dn, sn, bn);
  };
  if (!maps(&ly.in, &ly.out, w_in, w_out, n_experts)) return MOE_B200_ERR_TMA;
  if (n_shared > 0 && !maps(&ly.sh_in, &ly.sh_out, w_sh_in, w_sh_out, n_shared))
    return MOE_B200_ERR_TMA;
  ly.router_w = static_cast<const __nv_bfloat16*>(router_w);
  ly.bias = logit_bias;
  std::memcpy(static_cast<char*>(host_plan) + size_t(layer) * sizeof(StackLayer), &ly, sizeof(ly));
  return MOE_B200_OK;
}

int moe_b200_stack_infer(const void* plan, int32_t n_layers, const void* x, void* out,
                         int64_t n_tokens, int32_t d_model, int32_t d_hidden, int32_t n_experts,
                         int32_t n_shared, int32_t top_k, int32_t normalize, int32_t activation,
                         void* scratch, size_t scratch_bytes, int32_t* n_launches, int32_t* status,
                         void* stream) {
  StackShape o;
  if (n_layers < 1 || activation < 0 || activation > 4) return MOE_B200_ERR_SHAPE;
  const StackDevice& dev = stack_device();
  if (!stack_shape(dev, n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, &o))
    return MOE_B200_ERR_UNSUPPORTED;
  if (!plan || !x || !out || !scratch || !status) return MOE_B200_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(plan) & 63u) != 0 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) |
        reinterpret_cast<uintptr_t>(scratch)) & 15u) != 0)
    return MOE_B200_ERR_ALIGN;
  const StackScratch s = stack_scratch(scratch, n_tokens, d_model, n_shared, top_k);
  if (scratch_bytes < s.total) return MOE_B200_ERR_SCRATCH;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  launch_pdl(stack_reset_kernel, dim3(1), dim3(32), 0, st, s.ctr);
  StackArgs a{};
  a.layers = static_cast<const StackLayer*>(plan);
  a.n_layers = n_layers;
  a.T = int32_t(n_tokens);
  a.D = d_model;
  a.E = n_experts;
  a.S = n_shared;
  a.k = top_k;
  a.normalize = normalize;
  a.act = activation;
  a.n_stages = o.n_stages;
  a.router_extra = o.router_extra;
  a.out_boxes = d_model % 64 == 0 ? 1 : 2;
  a.kshift = top_k <= 8 ? 3 : 4;
  a.sh_tokens = o.sh_tokens;
  a.sh_blocks = o.sh_blocks;
  a.n_items = o.n_items;
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.out = static_cast<__nv_bfloat16*>(out);
  a.xbuf = s.xbuf;
  a.partial = s.partial;
  a.idx = s.idx;
  a.ctr = s.ctr;
  a.status = status;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(dev.grid()));
  cfg.blockDim = dim3(ST_THREADS);
  cfg.dynamicSmemBytes = size_t(o.smem);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // the CTAs wait on one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, n_experts <= 96 ? stack_kernel<3> : stack_kernel<8>, a);
  if (err != cudaSuccess) return MOE_B200_ERR_CUDA;
  if (n_launches) *n_launches = 2;
  return MOE_B200_OK;
}

}  // extern "C"
