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
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "../../include/moe_b200.h"
#include "act.cuh"
#include "pdl.cuh"
#include "ptx.cuh"
#include "routing.cuh"
#include "tma_map.cuh"

namespace moe {

constexpr int ST_H = 128;                  // hidden units per expert
constexpr int ST_SLICE = 32;               // of them in one work item
constexpr int ST_SLICES = ST_H / ST_SLICE;
constexpr int ST_STAGE = 8192;             // ring stage: [64 d x (32 gate + 32 up)] or [32 units x 128 d]
constexpr int ST_HALF = ST_STAGE / 2;      // one TMA box
// 8 warps: with one more (a warp of its own for the TMA loads) a thread is left with 168 registers, and
// the spills, which find no room in the L1 that 227 KB of shared memory leave, cost more than the work.
constexpr int ST_WARPS = 8;
constexpr int ST_THREADS = ST_WARPS * 32;
constexpr int ST_PASS = 16;                // tokens per pass over an item (two mma column tiles)
constexpr int ST_ACC_LD = 68;              // floats between tokens of the up accumulators
constexpr int ST_ACC_BYTES = 4 * ST_PASS * ST_ACC_LD * 4;
constexpr int ST_HID_LD = 40;              // bf16 between tokens of the hidden rows (80 B: no conflicts)
constexpr int ST_MAX_T = 256;
constexpr int ST_MAX_ITEMS = 8;            // items of one CTA and layer
constexpr int ST_MAX_STAGES = 24;
constexpr int ST_PARTS = 32;               // barriers for the two parts of an item; more than stages
constexpr int ST_MAX_SLOTS = 4;            // tokens of one CTA
// Router weight chunks (four columns of a row) that a thread holds across the hand-over, in registers;
// as many more as fit go to the row buffers, which are free then (all 45 at 76 experts and d_model
// 576). Loaded after the hand-over, they cost an L2 latency a batch.
constexpr int ST_ROUTER_PRE = 27;
static_assert(ST_MAX_ITEMS <= ST_WARPS, "a warp lists one item's tokens");

struct alignas(64) StackLayer {
  CUtensorMap in, out, sh_in, sh_out;
  const __nv_bfloat16* router_w;           // [D, E]
  const float* bias;                       // [E] or null
};

struct StackArgs {
  const StackLayer* layers;
  int32_t n_layers, T, D, E, S, k, normalize, act;
  int32_t n_stages;                        // of the ring
  int32_t xs_bufs;                         // token row buffers: 2 (the next pass's rows arrive under
                                           // this one's work) or 1
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
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async_8(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst_smem), "l"(src) : "memory");
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
__device__ __forceinline__ float stack_act(int act, float g) {
  switch (act) {
    case ACT_SILU: return act_f<ACT_SILU>(g);
    case ACT_GELU: return act_f<ACT_GELU>(g);
    case ACT_RELU: return act_f<ACT_RELU>(g);
    case ACT_SIGMOID: return act_f<ACT_SIGMOID>(g);
    default: return act_f<ACT_TANH>(g);
  }
}

// Shared memory behind the ring, in order.
struct StackSmem {
  int xs, acc, hid, list, xrow, res, tokw, lg, bars, misc, total;
};
__host__ __device__ inline StackSmem stack_smem(int T, int D, int n_stages, int xs_bufs) {
  const int dpad = (D + 63) / 64 * 64;
  StackSmem s;
  int at = n_stages * ST_STAGE;
  auto take = [&](int bytes) {
    const int r = at;
    at += (bytes + 15) / 16 * 16;
    return r;
  };
  s.xs = take(xs_bufs * ST_PASS * (dpad * 2 + 16));    // token rows of a pass
  s.acc = take(ST_ACC_BYTES);                          // up accumulators; token phase: partial sums
  s.hid = take((T + ST_PASS - 1) / ST_PASS * ST_PASS * ST_HID_LD * 2);
  s.list = take(2 * ST_MAX_ITEMS * T * 2);             // an item's tokens, and their pairs
  s.xrow = take(dpad * 4);                             // token phase: the row, fp32
  s.res = take(ST_MAX_SLOTS * D * 2);                  // residual rows of this CTA's tokens
  s.tokw = take(ST_MAX_SLOTS * 16 * 4);                // their pairs' weights
  s.lg = take(MAX_EXPERTS * 4);
  s.bars = take(ST_PARTS * 8);
  s.misc = take(16 + ST_MAX_ITEMS * 4 + ST_MAX_ITEMS * 16);   // abort flag, token counts, items
  s.total = at;
  return s;
}

// One warp: the k largest of lg[0, E) (value descending, ties to the lowest index) and their softmax
// weights, rounded to bf16. NS = ceil(E / 32) values per lane. Lane j returns the j-th choice.
template <int NS>
__device__ __forceinline__ void stack_select(const float* lg, int E, int k, int normalize, int lane,
                                             int* idx, float* weight) {
  float v[NS];
  uint32_t key[NS];
  float mx = -CUDART_INF_F;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const int e = i * 32 + lane;
    v[i] = e < E ? lg[e] : -CUDART_INF_F;
    const uint32_t fk = float_key(v[i]);
    key[i] = e < E ? (fk == 0u ? 1u : fk) : 0u;
    mx = fmaxf(mx, v[i]);
  }
  float denom = 0.f;
  if (!normalize) {
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
    for (int i = 0; i < NS; ++i) denom += i * 32 + lane < E ? expf(v[i] - mx) : 0.f;
#pragma unroll
    for (int o = 16; o; o >>= 1) denom += __shfl_xor_sync(0xffffffffu, denom, o);
  }
  int sel = 0;
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
  const bool active = lane < k;
  const float val = active ? lg[sel] : -CUDART_INF_F;
  float w;
  if (normalize) {
    const float top = __shfl_sync(0xffffffffu, val, 0);
    const float ex = active ? expf(val - top) : 0.f;
    float s = ex;
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    w = ex / s;
  } else {
    w = active ? expf(val - mx) / denom : 0.f;
  }
  *idx = active ? sel : 0xffff;
  *weight = active ? __bfloat162float(__float2bfloat16(w)) : 1.f;   // past k: the shared experts
}

__global__ void __launch_bounds__(ST_THREADS, 1) stack_kernel(const StackArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  const StackSmem L = stack_smem(p.T, p.D, p.n_stages, p.xs_bufs);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bars);   // [ST_PARTS] up / down weights of an item
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.misc);
  int* cnt = reinterpret_cast<int*>(smem + L.misc + 16);
  StackItem* items = reinterpret_cast<StackItem*>(smem + L.misc + 16 + ST_MAX_ITEMS * 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = int(gridDim.x), cta = int(blockIdx.x);
  const int D = p.D, dpad = (D + 63) / 64 * 64;
  const int n_in = dpad / 64, n_box = n_in, n_out = (n_box + 1) / 2;   // ring stages of one item
  const int NS = p.n_stages;
  const int kS = p.k + p.S;
  // this CTA's items (all but the last round are full)
  const int rounds = (p.n_items + G - 1) / G;
  const int n_mine = rounds - (stack_position(rounds - 1, cta, G) < p.n_items ? 0 : 1);

  if (tid == 0) {
    for (int s = 0; s < ST_PARTS; ++s) mbar_init(full + s, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (tid < n_mine) items[tid] = stack_item(p, stack_position(tid, cta, G));
  __syncthreads();
  pdl_wait();   // the counters, x and the weights may come from the kernels before this one

  // The ring is filled from where it is emptied: whenever an item's stages are free, one warp issues as
  // many of the coming loads as there is room for. (The loads' state lives in that warp.)
  constexpr int FILL_WARP = ST_WARPS - 1;
  const uint32_t ring_u = smem_u32(smem);
  int f_s = 0, f_free = NS, f_layer = 0, f_item = 0, f_stage = 0, f_part = 0;
  auto refill = [&](int freed) {
    f_free += freed;
    while (f_free > 0 && f_layer < p.n_layers && n_mine > 0) {
      const StackItem item = items[f_item];
      const StackLayer* ly = p.layers + f_layer;
      const bool shared = item.expert >= p.E, down = f_stage >= n_in;
      const int g = shared ? item.expert - p.E : item.expert;
      const int n = min(f_free, (down ? n_in + n_out : n_in) - f_stage);   // stages of this part
      uint64_t* bar = full + f_part % ST_PARTS;
      if (lane == 0 && f_stage == (down ? n_in : 0))
        mbar_expect_tx(bar, down ? n_box * ST_HALF : n_in * ST_STAGE);
      __syncwarp();
      const CUtensorMap* map = down ? (shared ? &ly->sh_out : &ly->out) : (shared ? &ly->sh_in : &ly->in);
      for (int i = lane; i < n; i += 32) {
        const int st = f_s + i < NS ? f_s + i : f_s + i - NS;
        uint8_t* dst = smem + st * ST_STAGE;
        if (down) {
          const int b = 2 * (f_stage - n_in + i);
          tma_load_3d(dst, map, bar, b * 64, item.slice * ST_SLICE, g);
          if (b + 1 < n_box) tma_load_3d(dst + ST_HALF, map, bar, b * 64 + 64, item.slice * ST_SLICE, g);
        } else {
          tma_load_3d(dst, map, bar, item.slice * ST_SLICE, (f_stage + i) * 64, g);
          tma_load_3d(dst + ST_HALF, map, bar, ST_H + item.slice * ST_SLICE, (f_stage + i) * 64, g);
        }
      }
      __syncwarp();
      f_s = f_s + n < NS ? f_s + n : f_s + n - NS;
      f_free -= n;
      f_stage += n;
      if (f_stage == n_in) ++f_part;
      if (f_stage == n_in + n_out) {
        ++f_part;
        f_stage = 0;
        if (++f_item == n_mine) {
          f_item = 0;
          ++f_layer;
        }
      }
    }
  };
  if (warp == FILL_WARP) refill(0);

  const uint32_t xs_ld = dpad * 2 + 16, xs_bytes = ST_PASS * xs_ld;
  float* acc_s = reinterpret_cast<float*>(smem + L.acc);
  __nv_bfloat16* hid_s = reinterpret_cast<__nv_bfloat16*>(smem + L.hid);
  uint16_t* list = reinterpret_cast<uint16_t*>(smem + L.list);   // [item][tokens | pairs][T]
  float* xrow = reinterpret_cast<float*>(smem + L.xrow);
  __nv_bfloat16* res = reinterpret_cast<__nv_bfloat16*>(smem + L.res);
  float* tokw = reinterpret_cast<float*>(smem + L.tokw);
  float* lg = reinterpret_cast<float*>(smem + L.lg);
  const int token_ctas = min(p.T, G);
  const bool has_token = cta < p.T;
  const int kpad = 1 << p.kshift;

  // One thread looks at the counter, the CTA follows. False: given up.
  auto grid_wait = [&](const uint32_t* ctr, uint32_t target) {
    if (tid == 0) {
      uint32_t n = 0;
      while (load_gpu(ctr) < target) {
        if (++n > (1u << 22) || ((n & 1023u) == 0 && *reinterpret_cast<volatile int32_t*>(p.status))) {
          atomicExch(p.status, ST_WAIT_TIMEOUT);
          *abort_flag = 1;
          break;
        }
      }
    }
    __syncthreads();
    if (*abort_flag == 0) return true;
    for (int n = 0; n < 1000; ++n) __nanosleep(1000);   // let the loads in flight land
    return false;
  };
  int ring_s = 0, part = 0;   // the ring as the consumers see it: the current item's first stage, its part
  auto part_wait = [&](int q) {
    if (!mbar_wait(full + q % ST_PARTS, (q / ST_PARTS) & 1, p.status)) {
      atomicExch(p.status, ST_WAIT_TIMEOUT);
      *abort_flag = 1;
    }
  };
  auto stage_of = [&](int c) {   // (an item may have more stages than the ring)
    int s = ring_s + c;
    while (s >= NS) s -= NS;
    return s;
  };
  auto item_done = [&] {
    ring_s = stage_of(n_in + n_out);
    part += 2;
  };

  // router weight: a thread owns four columns (4 * (tid % P)) of every Q-th row
  const int P = p.E / 4, Q = ST_THREADS / P;
  const int rp = tid % P, rq = tid / P;
  const int router_more =   // chunks of this thread in the row buffers
      max(0, min((D - rq + Q - 1) / Q - ST_ROUTER_PRE, int(p.xs_bufs * xs_bytes / (ST_THREADS * 8))));
  const int cg = D / 4;   // token phase: 16-byte column groups
  const __nv_bfloat16* rw = p.layers[0].router_w;   // (the next layer's are fetched a layer ahead)
  const float* bias = p.layers[0].bias;

  for (int l = 0; l <= p.n_layers; ++l) {
    const bool last = l == p.n_layers;
    // ------------------------------------------------------------------ token phase
    if (has_token) {
      uint2 wr[ST_ROUTER_PRE];   // (on its way while this CTA waits for the others' partial rows)
#pragma unroll
      for (int i = 0; i < ST_ROUTER_PRE; ++i) {
        const int d = rq + i * Q;
        wr[i] = !last && rq < Q && d < D
                    ? __ldg(reinterpret_cast<const uint2*>(rw + d * p.E + 4 * rp))
                    : make_uint2(0u, 0u);
      }
      if (!last && rq < Q) {
        const __nv_bfloat16* src = rw + (rq + ST_ROUTER_PRE * Q) * p.E + 4 * rp;
        for (int i = 0; i < router_more; ++i)
          cp_async_8(smem_u32(smem + L.xs) + (i * ST_THREADS + tid) * 8, src + i * Q * p.E);
      }
      cp_async_commit();
      if (l > 0 && !grid_wait(p.ctr + 1, uint32_t(l) * G)) return;
      for (int t = cta, slot = 0; t < p.T; t += G, ++slot) {
        __nv_bfloat16* my_res = res + slot * D;
        float* my_w = tokw + slot * 16;
        // the row: residual + the pairs' partial rows, in order; four columns per thread and step,
        // the rows cut into `groups` interleaved sets when there are threads for it
        const int groups = max(1, ST_THREADS / cg);
        if (l > 0) {
          const int R = kS * ST_SLICES;
          const float* base = p.partial + int64_t(t) * R * D;
          for (int i = tid; i < groups * cg; i += ST_THREADS) {
            const int g = i / cg, c = i - g * cg;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int r0 = g; r0 < R; r0 += 16 * groups) {
              float4 v[16];
#pragma unroll
              for (int u = 0; u < 16; ++u) {
                const int r = r0 + u * groups;
                v[u] = r < R ? ldcg4(base + r * D + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
              }
#pragma unroll
              for (int u = 0; u < 16; ++u) {
                const int r = r0 + u * groups;
                const float w = r < R ? my_w[r / ST_SLICES] : 0.f;
                a.x += w * v[u].x;
                a.y += w * v[u].y;
                a.z += w * v[u].z;
                a.w += w * v[u].w;
              }
            }
            *reinterpret_cast<float4*>(acc_s + g * D + 4 * c) = a;
          }
          __syncthreads();
        }
        for (int d = 2 * tid; d < dpad; d += 2 * ST_THREADS) {
          float v0 = 0.f, v1 = 0.f;
          if (d < D) {
            __nv_bfloat162 h;
            if (l > 0) {
              const float2 f = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(my_res + d));
              v0 = f.x;
              v1 = f.y;
              for (int g = 0; g < groups; ++g) {
                v0 += acc_s[g * D + d];
                v1 += acc_s[g * D + d + 1];
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
          xrow[d] = v0;
          xrow[d + 1] = v1;
        }
        __syncthreads();
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
          for (int i = 0; i < ST_ROUTER_PRE; ++i) {
            const int d = rq + i * Q;
            if (d < D) add(wr[i], xrow[d]);
          }
          cp_async_wait<0>();   // (a thread reads back what it copied itself)
          const uint2* ws = reinterpret_cast<const uint2*>(smem + L.xs) + tid;
#pragma unroll 4
          for (int i = 0; i < router_more; ++i) add(ws[i * ST_THREADS], xrow[rq + (ST_ROUTER_PRE + i) * Q]);
          for (int d0 = rq + (ST_ROUTER_PRE + router_more) * Q; d0 < D; d0 += 16 * Q) {
            uint2 w[16];
#pragma unroll
            for (int i = 0; i < 16; ++i)
              w[i] = d0 + i * Q < D ? __ldg(reinterpret_cast<const uint2*>(
                                          rw + (d0 + i * Q) * p.E + 4 * rp))
                                    : make_uint2(0u, 0u);
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (d0 + i * Q < D) add(w[i], xrow[d0 + i * Q]);
          }
          *reinterpret_cast<float4*>(acc_s + rq * p.E + 4 * rp) = make_float4(a0, a1, a2, a3);
        }
        const float b = bias != nullptr && tid < p.E ? __ldg(bias + tid) : 0.f;
        __syncthreads();
        if (tid < p.E) {   // (at most 256 experts: one thread each)
          float s = 0.f;
#pragma unroll 16
          for (int q = 0; q < Q; ++q) s += acc_s[q * p.E + tid];
          lg[tid] = __bfloat162float(__float2bfloat16(s)) + b;
        }
        __syncthreads();
        if (warp == 0) {
          int sel;
          float w;
          if (p.E <= 32) stack_select<1>(lg, p.E, p.k, p.normalize, lane, &sel, &w);
          else if (p.E <= 64) stack_select<2>(lg, p.E, p.k, p.normalize, lane, &sel, &w);
          else if (p.E <= 96) stack_select<3>(lg, p.E, p.k, p.normalize, lane, &sel, &w);
          else if (p.E <= 128) stack_select<4>(lg, p.E, p.k, p.normalize, lane, &sel, &w);
          else stack_select<8>(lg, p.E, p.k, p.normalize, lane, &sel, &w);
          if (lane < kpad) p.idx[t * kpad + lane] = uint16_t(sel);
          if (lane < kS) my_w[lane] = w;
        }
        __syncthreads();
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
        for (int i = lane; i < item.n; i += 32) {
          tok[i] = uint16_t(item.t0 + i);
          pair[i] = uint16_t((item.t0 + i) * kS + p.k + (item.expert - p.E));
        }
        n = item.n;
      } else {
        for (int b = lane * 8; b - lane * 8 < p.T * kpad; b += 256) {
          uint4 v = make_uint4(~0u, ~0u, ~0u, ~0u);
          if (b < p.T * kpad) v = __ldcg(reinterpret_cast<const uint4*>(p.idx + b));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
          uint32_t hits = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            hits |= uint32_t((w[i] & 0xffffu) == uint32_t(item.expert)) << (2 * i);
            hits |= uint32_t((w[i] >> 16) == uint32_t(item.expert)) << (2 * i + 1);
          }
          // a token chooses an expert once; eight entries are one token's (or half of one's)
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
    __syncthreads();
    // the rows of the tokens [n0, n0 + 16) of item r, into row buffer `buf`
    auto gather = [&](int r, int n0, int buf) {
      const uint16_t* tok = list + 2 * r * p.T + n0;
      const int nn = min(ST_PASS, cnt[r] - n0), cpr = dpad / 8;
      const uint32_t dst = smem_u32(smem + L.xs) + buf * xs_bytes;
      for (int row = warp; row < nn; row += ST_WARPS) {
        const __nv_bfloat16* src = p.xbuf + int64_t(tok[row]) * D;
        for (int c = lane; c < cpr; c += 32)
          cp_async_16(dst + row * xs_ld + c * 16, c * 8 < D ? src + c * 8 : src, c * 8 < D ? 16u : 0u);
      }
      cp_async_commit();
    };
    // the rows of the pass after (r, n0): the same item's next tokens, or the next item that has any
    auto gather_next = [&](int r, int n0, int buf) {
      n0 += ST_PASS;
      if (r < 0 || n0 >= cnt[r]) {
        n0 = 0;
        do ++r;
        while (r < n_mine && cnt[r] == 0);
      }
      if (r < n_mine) gather(r, n0, buf);
    };
    int buf = 0;
    gather_next(-1, 0, 0);
    for (int r = 0; r < n_mine; ++r) {
      const int slice = items[r].slice;
      const int n = cnt[r];
      if (n == 0) {   // nobody chose it: the ring moves on
        if (warp == FILL_WARP) {
          part_wait(part);
          refill(n_in);
          part_wait(part + 1);
          refill(n_out);
        }
        item_done();
        continue;
      }
      // up/gate + GLU: 64 outputs (gate and up, two mma rows each) x 16 tokens; warps 2i, 2i + 1 take
      // the i-th quarter of every 64-deep stage
      const int mg = warp & 1, kp = warp >> 1;
      for (int n0 = 0; n0 < n; n0 += ST_PASS) {
        const int nn = min(ST_PASS, n - n0);
        cp_async_wait<0>();
        __syncthreads();
        if (p.xs_bufs == 2) gather_next(r, n0, buf ^ 1);   // (under this pass's work)
        if (n0 == 0) part_wait(part);
        float acc[2][2][4] = {};
        const int a_k = kp * 16 + (lane & 7) + ((lane >> 4) & 1) * 8;
        const int a_c = (lane >> 3) & 1;
        const uint32_t sw = (a_k >> 1) & 3;
        const uint32_t a0 = mg * ST_HALF + a_k * 64 + ((a_c ^ sw) << 4);
        const uint32_t a1 = mg * ST_HALF + a_k * 64 + (((a_c + 2) ^ sw) << 4);
        uint32_t b_addr = smem_u32(smem + L.xs) + buf * xs_bytes + (kp * 16 + ((lane >> 3) & 1) * 8) * 2;
        int s = ring_s;
        if (nn > 8) {
          b_addr += ((lane & 7) + ((lane >> 4) & 1) * 8) * xs_ld;
#pragma unroll 3
          for (int c = 0; c < n_in; ++c) {
            uint32_t a[2][4], b[4];
            ldsm4_t(ring_u + s * ST_STAGE + a0, a[0]);
            ldsm4_t(ring_u + s * ST_STAGE + a1, a[1]);
            ldsm4(b_addr + c * 128, b);
            mma_bf16(acc[0][0], a[0], b[0], b[1]);
            mma_bf16(acc[1][0], a[1], b[0], b[1]);
            mma_bf16(acc[0][1], a[0], b[2], b[3]);
            mma_bf16(acc[1][1], a[1], b[2], b[3]);
            if (++s == NS) s = 0;
          }
        } else {
          b_addr += (lane & 7) * xs_ld;
#pragma unroll 3
          for (int c = 0; c < n_in; ++c) {
            uint32_t a[2][4], b[2];
            ldsm4_t(ring_u + s * ST_STAGE + a0, a[0]);
            ldsm4_t(ring_u + s * ST_STAGE + a1, a[1]);
            ldsm2(b_addr + c * 128, b);
            mma_bf16(acc[0][0], a[0], b[0], b[1]);
            mma_bf16(acc[1][0], a[1], b[0], b[1]);
            if (++s == NS) s = 0;
          }
        }
        float* dst = acc_s + (kp * ST_PASS + 2 * (lane & 3)) * ST_ACC_LD + mg * 32 + (lane >> 2);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (q == 1 && nn <= 8) break;
            float* d = dst + 8 * q * ST_ACC_LD + m * 16;
            d[0] = acc[m][q][0];
            d[ST_ACC_LD] = acc[m][q][1];
            d[8] = acc[m][q][2];
            d[ST_ACC_LD + 8] = acc[m][q][3];
          }
        __syncthreads();
        if (n0 + ST_PASS >= n && warp == FILL_WARP) refill(n_in);
        if (p.xs_bufs == 1)
          gather_next(r, n0, 0);
        else
          buf ^= 1;
        for (int row = warp; row < nn; row += ST_WARPS) {   // 32 units of a token per warp
          float g = 0.f, up = 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            g += acc_s[(q * ST_PASS + row) * ST_ACC_LD + lane];
            up += acc_s[(q * ST_PASS + row) * ST_ACC_LD + 32 + lane];
          }
          hid_s[(n0 + row) * ST_HID_LD + lane] = __float2bfloat16(stack_act(p.act, g) * up);
        }
      }
      __syncthreads();
      // down: D outputs in rows of 16, 32 deep; a warp takes every 8th row
      part_wait(part + 1);
      const uint16_t* pair = list + (2 * r + 1) * p.T;
      const int u0 = (lane & 7) + ((lane >> 4) & 1) * 8, c0 = (lane >> 3) & 1;
      for (int n0 = 0; n0 < n; n0 += ST_PASS) {
        uint32_t b[2][4];
        const uint32_t h_addr = smem_u32(hid_s) +
                                (n0 + (lane & 7) + ((lane >> 4) & 1) * 8) * (ST_HID_LD * 2) +
                                ((lane >> 3) & 1) * 16;
        ldsm4(h_addr, b[0]);
        ldsm4(h_addr + 32, b[1]);
        float* dst[4];   // this thread's four tokens
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = n0 + 8 * (q >> 1) + 2 * (lane & 3) + (q & 1);
          dst[q] = i < n ? p.partial + (int64_t(pair[i]) * ST_SLICES + slice) * D + (lane >> 2)
                         : nullptr;
        }
        const bool two = n - n0 > 8;
#pragma unroll 2
        for (int m = warp; m < D / 16; m += ST_WARPS) {
          uint32_t a[2][4];
          const uint32_t box = ring_u + stage_of(n_in + (m >> 3)) * ST_STAGE + ((m >> 2) & 1) * ST_HALF;
          const uint32_t ch = (((m & 3) * 2 + c0) ^ (u0 & 7)) << 4;
          ldsm4_t(box + u0 * 128 + ch, a[0]);
          ldsm4_t(box + (u0 + 16) * 128 + ch, a[1]);
          float acc[2][4] = {};
          mma_bf16(acc[0], a[0], b[0][0], b[0][1]);
          mma_bf16(acc[0], a[1], b[1][0], b[1][1]);
          if (two) {
            mma_bf16(acc[1], a[0], b[0][2], b[0][3]);
            mma_bf16(acc[1], a[1], b[1][2], b[1][3]);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (dst[q] != nullptr) {
              dst[q][m * 16] = acc[q >> 1][q & 1];
              dst[q][m * 16 + 8] = acc[q >> 1][2 + (q & 1)];
            }
        }
      }
      __syncthreads();
      if (warp == FILL_WARP) refill(n_out);
      item_done();
    }
    if (tid == 0) arrive_gpu(p.ctr + 1);
  }
}

// ---------------------------------------------------------------------------------- host
static int stack_grid() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
  }
  return n;
}

__global__ void stack_reset_kernel(uint32_t* ctr) {
  pdl_wait();
  if (threadIdx.x < 2) ctr[threadIdx.x] = 0u;
}

// The shape side of a launch; false: the layer-by-layer path is the one that takes it.
struct StackShape {
  int sh_tokens, sh_blocks, n_items, n_stages, xs_bufs, smem;
};
static bool stack_shape(int64_t T, int D, int H, int E, int S, int k, StackShape* o) {
  if (T < 1 || T > ST_MAX_T || H != ST_H || D < 64 || D % 32 != 0 || D > 1024 || E < 4 ||
      E % 4 != 0 || S < 0 || E + S > MAX_EXPERTS || k < 1 || k > E || k + S > 16)
    return false;
  const int grid = stack_grid();
  if (T > int64_t(ST_MAX_SLOTS) * grid) return false;
  // a shared expert sees every token: 32 of them per work item keep it in the range of the others
  o->sh_tokens = int(std::min<int64_t>(T, 32));
  o->sh_blocks = int((T + o->sh_tokens - 1) / o->sh_tokens);
  o->n_items = ST_SLICES * (E + S * o->sh_blocks);
  if (o->n_items > ST_MAX_ITEMS * grid) return false;
  // two row buffers unless they cost the ring the stages that an item's up weights need at once
  const int limit = 232448 - 1024, n_in = (D + 63) / 64;
  for (o->xs_bufs = 2; o->xs_bufs > 0; --o->xs_bufs) {
    const int rest = stack_smem(int(T), D, 0, o->xs_bufs).total;
    o->n_stages = std::min((limit - rest) / ST_STAGE, ST_MAX_STAGES);
    if (limit > rest && o->n_stages >= n_in) break;
  }
  if (o->xs_bufs == 0) return false;
  o->smem = stack_smem(int(T), D, o->n_stages, o->xs_bufs).total + 1024;
  return true;
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
  return stack_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, &o) ? 1 : 0;
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
    const uint64_t di[3] = {uint64_t(2 * d_hidden), uint64_t(d_model), uint64_t(g)};
    const uint64_t si[2] = {uint64_t(4 * d_hidden), uint64_t(4 * d_hidden) * d_model};
    const uint32_t bi[3] = {ST_SLICE, 64, 1};
    const uint64_t dn[3] = {uint64_t(d_model), uint64_t(d_hidden), uint64_t(g)};
    const uint64_t sn[2] = {uint64_t(2 * d_model), uint64_t(2 * d_model) * d_hidden};
    const uint32_t bn[3] = {64, ST_SLICE, 1};
    return make_map(in, wi, 3, di, si, bi, CU_TENSOR_MAP_SWIZZLE_64B) &&
           make_map(out, wo, 3, dn, sn, bn);
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
  if (!stack_shape(n_tokens, d_model, d_hidden, n_experts, n_shared, top_k, &o))
    return MOE_B200_ERR_UNSUPPORTED;
  if (!plan || !x || !out || !scratch || !status) return MOE_B200_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(plan) & 63u) != 0 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) |
        reinterpret_cast<uintptr_t>(scratch)) & 15u) != 0)
    return MOE_B200_ERR_ALIGN;
  const StackScratch s = stack_scratch(scratch, n_tokens, d_model, n_shared, top_k);
  if (scratch_bytes < s.total) return MOE_B200_ERR_SCRATCH;
  static std::once_flag once;
  static cudaError_t attr_err = cudaSuccess;
  std::call_once(once, [] {
    attr_err = cudaFuncSetAttribute(stack_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
  });
  if (attr_err != cudaSuccess) return MOE_B200_ERR_CUDA;
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
  a.xs_bufs = o.xs_bufs;
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
  cfg.gridDim = dim3(unsigned(stack_grid()));
  cfg.blockDim = dim3(ST_THREADS);
  cfg.dynamicSmemBytes = size_t(o.smem);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // the CTAs wait on one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, stack_kernel, a) != cudaSuccess) return MOE_B200_ERR_CUDA;
  if (n_launches) *n_launches = 2;
  return MOE_B200_OK;
}

}  // extern "C"
