// Muon's step on stacked expert weights (src/train/optim.py:75-105) in three launches over all of
// them: momentum and Nesterov direction with the directions' norms; the Newton-Schulz iteration of
// every matrix inside one CTA; the weight update with both norms. 78 experts of [576, 256] and
// [128, 576]: 168 us; as torch operations around 26 launches of the grouped GEMMs per stack 2040 us,
// of which the element-wise operations (13 passes over the weights) 1.2 ms.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "../../include/moe_b200.h"
#include "gemm.cuh"
#include "tma_map.cuh"

namespace moe {

constexpr int MU_THREADS = 256;
constexpr int MU_MAX = 16;          // tensors per launch
constexpr int MU_PARTS = 32;        // partial norms per matrix at most

struct MuonTensor {
  const uint4* grad;
  uint4* buf;
  uint4* dir;
  void* p;
  float* sumsq;          // [groups, parts] partial |dir|^2
  int64_t first_block;   // of this tensor in the launch
  int32_t groups, parts, pieces, p_is_fp32;   // pieces: 16-byte pieces of one matrix
  float step;
};
struct MuonTensors {
  MuonTensor t[MU_MAX];
  int32_t n;
};

__device__ __forceinline__ void unpack8(const uint4& r, float* f) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16(v)); }
// torch.lerp's two forms (the one with the smaller weight on the difference)
__device__ __forceinline__ float lerp_like_torch(float a, float b, float w) {
  return w < 0.5f ? a + w * (b - a) : b - (b - a) * (1.f - w);
}
__device__ __forceinline__ float block_sum(float v) {
  __shared__ float part[MU_THREADS / 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < MU_THREADS / 32; ++i) t += part[i];
  return t;
}
__device__ __forceinline__ const MuonTensor& muon_tensor(const MuonTensors& ts, int64_t block) {
  int i = 0;
  while (i + 1 < ts.n && ts.t[i + 1].first_block <= block) ++i;
  return ts.t[i];
}

// buf <- lerp(buf, grad, w_grad); dir = lerp(grad, buf, momentum), both rounded to bf16 as the
// operations one by one do, and a part of |dir|^2 of the matrix per block (no atomics: the norm is
// the same from run to run). HBM-bound: 8 bytes per value (grad and buf read, buf and dir written).
__global__ void __launch_bounds__(MU_THREADS)
    muon_direction_kernel(const __grid_constant__ MuonTensors ts, float w_grad, float momentum,
                          float* norms) {
  pdl_trigger();
  pdl_wait();
  if (norms != nullptr && blockIdx.x == 0 && threadIdx.x < 3) norms[threadIdx.x] = 0.f;
  const MuonTensor& t = muon_tensor(ts, blockIdx.x);
  const int32_t local = int32_t(blockIdx.x - t.first_block);
  const int32_t group = local / t.parts, part = local % t.parts;
  const int64_t base = int64_t(group) * t.pieces;
  float ss = 0.f;
  for (int i = part * MU_THREADS + threadIdx.x; i < t.pieces; i += t.parts * MU_THREADS) {
    float g[8], b[8];
    unpack8(__ldcs(t.grad + base + i), g);
    unpack8(__ldcs(t.buf + base + i), b);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      b[k] = round_bf16(lerp_like_torch(b[k], g[k], w_grad));
      g[k] = round_bf16(lerp_like_torch(g[k], b[k], momentum));
      ss += g[k] * g[k];
    }
    __stcs(t.buf + base + i, pack8(b));
    t.dir[base + i] = pack8(g);
  }
  ss = block_sum(ss);
  if (threadIdx.x == 0) t.sumsq[local] = ss;
}

// delta = step * upd, p <- p * decay + delta, each rounded to p's type as the operations one by one
// do; norms[0] += |delta|^2, norms[1] += |p|^2, summed by the last block to finish in block order
// (norms[2] is its ticket). HBM-bound: 6 bytes per value in bf16.
__global__ void __launch_bounds__(MU_THREADS)
    muon_apply_kernel(const __grid_constant__ MuonTensors ts, float decay,
                      float* partials, float* norms) {
  pdl_trigger();
  pdl_wait();
  const MuonTensor& t = muon_tensor(ts, blockIdx.x);
  const int32_t local = int32_t(blockIdx.x - t.first_block);
  const int64_t base = int64_t(local / t.parts) * t.pieces;
  const float step = t.step;
  float dd = 0.f, pp = 0.f;
  for (int i = (local % t.parts) * MU_THREADS + threadIdx.x; i < t.pieces;
       i += t.parts * MU_THREADS) {
    float u[8], p[8];
    unpack8(__ldcs(t.dir + base + i), u);
    if (t.p_is_fp32) {
      float4* q = static_cast<float4*>(t.p) + 2 * (base + i);
      const float4 lo = __ldcs(q), hi = __ldcs(q + 1);
      const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        u[k] = u[k] * step;
        p[k] = v[k] * decay + u[k];
      }
      q[0] = make_float4(p[0], p[1], p[2], p[3]);
      q[1] = make_float4(p[4], p[5], p[6], p[7]);
    } else {
      uint4* q = static_cast<uint4*>(t.p) + base + i;
      unpack8(__ldcs(q), p);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        u[k] = round_bf16(u[k] * step);
        p[k] = round_bf16(round_bf16(p[k] * decay) + u[k]);
      }
      *q = pack8(p);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      dd += u[k] * u[k];
      pp += p[k] * p[k];
    }
  }
  dd = block_sum(dd);
  pp = block_sum(pp);
  __shared__ uint32_t ticket;
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = dd;
    partials[2 * blockIdx.x + 1] = pp;
    __threadfence();
    ticket = atomicInc(reinterpret_cast<uint32_t*>(norms + 2), gridDim.x - 1);
  }
  __syncthreads();
  if (ticket != gridDim.x - 1) return;
  __threadfence();
  dd = pp = 0.f;
  for (int i = threadIdx.x; i < int(gridDim.x); i += MU_THREADS) {
    dd += __ldcg(partials + 2 * i);
    pp += __ldcg(partials + 2 * i + 1);
  }
  dd = block_sum(dd);
  pp = block_sum(pp);
  if (threadIdx.x == 0) {
    norms[0] += dd;
    norms[1] += pp;
  }
}

// ------------------------------------------------------------------------- Newton-Schulz iteration
// X <- a X + (b A + c A A) X, A the Gram matrix of the short side, from X = dir / (|dir| + eps); one
// CTA runs all iterations of one matrix, which is either
//   wide  [128, n]:  A = X X^T (128 x 128), or
//   tall  [n, 256]:  A = X^T X (256 x 256, its blocks 00, 01, 11: it is symmetric).
// The long side is cut into tiles of 128, each [64 columns x 128 rows] boxes of 16 KB in the 128-byte
// swizzle, which UMMA reads K-major as well as MN-major: one copy of a tile serves the Gram product
// (contraction over the long side) and the update (contraction over the short one). A, then
// b A + c A A over it, stay in shared memory, the products in TMEM. A slot of shared memory per tile
// (t mod slots): six 32 KB slots hold a wide matrix up to n = 768 for all iterations; a tall one streams
// through two 64 KB slots from L2, the Gram pass upwards and the update pass downwards, so that each
// starts with the two tiles the other left. The normalisation is a factor of the first iteration (s^2 on
// its A, s on its result).
// What bounds it: the tensor pipe and its operand reads from shared memory; per tall iteration at
// n = 576 2.6 us of Gram, 1.6 us of A A and 5.4 us of update MMAs at full rate.
// Warps: 0 copies tiles in and out, 1 issues MMAs, 2..17 convert accumulators.
constexpr int NS_EPI_WARPS = 16;
constexpr int NS_THREADS = 64 + 32 * NS_EPI_WARPS;
constexpr uint32_t NS_BOX = 16384;
constexpr int NS_MAX_SLOTS = 6;
constexpr int NS_POLY_OFFSET_TALL = 2 * 4 * int(NS_BOX), NS_POLY_OFFSET_WIDE = 6 * 2 * int(NS_BOX);
constexpr int NS_DATA_BYTES = 14 * int(NS_BOX);
static_assert(NS_POLY_OFFSET_TALL + 6 * int(NS_BOX) == NS_DATA_BYTES, "two tiles, three blocks");
static_assert(NS_POLY_OFFSET_WIDE + 2 * int(NS_BOX) == NS_DATA_BYTES, "six tiles, one block");

struct NsBars {
  uint64_t full[NS_MAX_SLOTS];       // a tile has landed
  uint64_t gram_read[NS_MAX_SLOTS];  // the Gram MMAs have read a tile
  uint64_t acc_full;                 // A, then A A, complete in TMEM
  uint64_t conv_done;                // ... and converted into shared memory
  uint64_t upd_full[2];              // the product of an update is complete in TMEM half 0 / 1
  uint64_t upd_done[2];              // ... and its tile updated in shared memory
  uint64_t drain;
  uint32_t tmem;
};
constexpr int NS_SMEM = NS_DATA_BYTES + int(sizeof(NsBars)) + 1024;
static_assert(NS_SMEM <= 232448, "one CTA's shared memory");

struct NsJob {
  CUtensorMap map;      // [columns, rows, matrices], boxes of 64 x 128
  const float* sumsq;   // [matrices, parts]
  int32_t first_block, parts, length, tall;   // length: the long side
};
struct NsJobs {
  NsJob job[MU_MAX];
  int32_t n, steps;
  float a, b, c, eps;
  int32_t* status;
};

template <int K>
__device__ __forceinline__ void bulk_wait_done() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(K) : "memory");
}

template <bool TALL>
struct Ns {
  static constexpr int BOXES = TALL ? 4 : 2;
  static constexpr int SLOTS = TALL ? 2 : 6;
  static constexpr uint32_t TILE_BYTES = BOXES * NS_BOX;
  static constexpr int BLOCKS = TALL ? 3 : 1;      // 128 x 128 blocks of A
  static constexpr int POLY = TALL ? NS_POLY_OFFSET_TALL : NS_POLY_OFFSET_WIDE;
  static constexpr uint32_t UPD_COLS = TALL ? 256 : 128;

  // operands of 128 (or with N = 256 four boxes of) elements: K-major = 64 k per box, MN-major = 64
  // elements per box and one k per row
  static __device__ __forceinline__ uint64_t k_major(uint32_t base, int k16) {
    return umma_desc(base + uint32_t(k16 >> 2) * NS_BOX + uint32_t(k16 & 3) * 32u, 16, 1024);
  }
  static __device__ __forceinline__ uint64_t mn_major(uint32_t base, int k16) {
    return umma_desc(base + uint32_t(k16) * 2048u, NS_BOX, 1024);
  }

  static __device__ void copies(const NsJob& job, const NsJobs& js, int group, uint8_t* smem,
                                NsBars* bars) {
    const int nt = (job.length + 127) / 128;
    uint32_t loads = 0, in_flight = 0;
    bool ok = true;
    auto load = [&](int t) {
      const int s = t % SLOTS;
      mbar_expect_tx(bars->full + s, TILE_BYTES);
#pragma unroll 1
      for (int b = 0; b < BOXES; ++b)
        tma_load_3d(smem + s * TILE_BYTES + b * NS_BOX, &job.map, bars->full + s,
                    TALL ? 64 * b : 128 * t + 64 * b, TALL ? 128 * t : 0, group);
      loads ^= 1u << s;
      in_flight |= 1u << s;
    };
    for (int i = 0; i < js.steps && ok; ++i) {
      for (int t = 0; t < nt && ok; ++t) {
        if (i > 0 && t < SLOTS) continue;
        const int s = t % SLOTS;
        // the commits this slot has seen when its last tile has been read
        const int commits = i * ((nt - s + SLOTS - 1) / SLOTS) + t / SLOTS;
        if (t >= SLOTS) ok = mbar_wait(bars->gram_read + s, uint32_t(commits - 1) & 1u, js.status);
        if (ok) load(t);
      }
      const bool out = nt > SLOTS || i == js.steps - 1;
      for (int j = 0; j < nt && ok; ++j) {
        const int t = nt - 1 - j, v = i * nt + j;
        ok = mbar_wait(bars->upd_done + (v & 1), uint32_t(v >> 1) & 1u, js.status);
        if (!ok || !out) continue;
#pragma unroll 1
        for (int b = 0; b < BOXES; ++b)
          if (TALL || 128 * t + 64 * b < job.length)
            tma_store_3d(&job.map, smem + (t % SLOTS) * TILE_BYTES + b * NS_BOX,
                         TALL ? 64 * b : 128 * t + 64 * b, TALL ? 128 * t : 0, group);
        bulk_commit();
        if (j + SLOTS < nt) {
          bulk_wait_read<0>();
          load(t - SLOTS);
        }
      }
      // the next pass reads what these stores wrote
      bulk_wait_done<0>();
      asm volatile("fence.proxy.async;" ::: "memory");
    }
    if (!ok) atomicExch(js.status, ST_WAIT_TIMEOUT);
    for (int s = 0; s < SLOTS; ++s)   // nothing may still be landing when the CTA leaves
      if (in_flight >> s & 1u) {
        for (uint32_t n = 0; n < MOE_WAIT_LIMIT; ++n)
          if (mbar_try_wait(bars->full + s, (loads >> s & 1u) ^ 1u)) break;
      }
  }

  static __device__ void mmas(const NsJob& job, const NsJobs& js, uint32_t tiles, uint32_t poly,
                              uint32_t tmem, NsBars* bars) {
    const int nt = (job.length + 127) / 128;
    constexpr uint32_t KK = umma_idesc(128, 128, false, false);
    constexpr uint32_t KM = umma_idesc(128, 128, false, true);
    constexpr uint32_t MM = umma_idesc(128, 128, true, true);
    uint32_t loads = 0;
    bool ok = true;
    auto tile = [&](int t, bool loaded) {      // waits until tile t is there
      const int s = t % SLOTS;
      if (loaded) loads ^= 1u << s;
      ok = ok && mbar_wait(bars->full + s, (loads >> s & 1u) ^ 1u, js.status);
      tc_fence_after();
      return tiles + uint32_t(s) * TILE_BYTES;
    };
    auto done = [&](int v) {                   // update v has left TMEM and is in its tile
      if (v >= 0) ok = ok && mbar_wait(bars->upd_done + (v & 1), uint32_t(v >> 1) & 1u, js.status);
    };
    for (int i = 0; i < js.steps && ok; ++i) {
      done(i * nt - 2);
      done(i * nt - 1);
      tc_fence_after();
      for (int t = 0; t < nt && ok; ++t) {
        const uint32_t x = tile(t, i == 0 || t >= SLOTS);
        if (!ok) break;
        const int steps16 = min(8, (job.length - 128 * t) / 16);
#pragma unroll 1
        for (int k = 0; k < steps16; ++k) {
          const uint32_t acc = (t | k) ? 1u : 0u;
          if constexpr (TALL) {
            umma_f16(tmem, mn_major(x, k), mn_major(x, k), umma_idesc(128, 256, true, true), acc);
            umma_f16(tmem + 256, mn_major(x + 2 * NS_BOX, k), mn_major(x + 2 * NS_BOX, k), MM, acc);
          } else {
            umma_f16(tmem, k_major(x, k), k_major(x, k), KK, acc);
          }
        }
        umma_commit(bars->gram_read + t % SLOTS);
      }
      if (!ok) break;
      umma_commit(&bars->acc_full);
      ok = mbar_wait(&bars->conv_done, 0, js.status);
      if (!ok) break;
      tc_fence_after();
      // A A; block 10 is block 01 read along its columns
#pragma unroll 1
      for (int k = 0; k < 8; ++k) {
        const uint32_t acc = k ? 1u : 0u;
        const uint64_t a00 = k_major(poly, k);
        umma_f16(tmem, a00, a00, KK, acc);
        if constexpr (TALL) {
          const uint64_t a10 = mn_major(poly + 2 * NS_BOX, k);
          umma_f16(tmem + 128, a00, a10, KM, acc);
          umma_f16(tmem + 256, a10, a10, MM, acc);
        }
      }
      if constexpr (TALL) {
#pragma unroll 1
        for (int k = 0; k < 8; ++k) {
          const uint64_t a01 = k_major(poly + 2 * NS_BOX, k), a11 = k_major(poly + 4 * NS_BOX, k);
          umma_f16(tmem, a01, a01, KK, 1u);
          umma_f16(tmem + 128, a01, a11, KK, 1u);
          umma_f16(tmem + 256, a11, a11, KK, 1u);
        }
      }
      umma_commit(&bars->acc_full);
      ok = mbar_wait(&bars->conv_done, 1, js.status);
      tc_fence_after();
      for (int j = 0; j < nt && ok; ++j) {
        const int t = nt - 1 - j, v = i * nt + j;
        const uint32_t x = tile(t, j >= SLOTS);
        done(v - 2);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem + uint32_t(v & 1) * UPD_COLS;
        if constexpr (TALL) {
#pragma unroll 1
          for (int k = 0; k < 8; ++k) {
            const uint64_t xk = k_major(x, k);
            umma_f16(d, xk, k_major(poly, k), KK, k ? 1u : 0u);
            umma_f16(d + 128, xk, mn_major(poly + 2 * NS_BOX, k), KM, k ? 1u : 0u);
          }
#pragma unroll 1
          for (int k = 0; k < 8; ++k) {
            const uint64_t xk = k_major(x + 2 * NS_BOX, k);
            umma_f16(d, xk, k_major(poly + 2 * NS_BOX, k), KK, 1u);
            umma_f16(d + 128, xk, k_major(poly + 4 * NS_BOX, k), KK, 1u);
          }
        } else {
          const uint32_t n = uint32_t(min(128, job.length - 128 * t));
          const uint32_t idesc = umma_idesc(128, 0, false, true) | (n >> 3) << 17;
#pragma unroll 1
          for (int k = 0; k < 8; ++k)
            umma_f16(d, k_major(poly, k), mn_major(x, k), idesc, k ? 1u : 0u);
        }
        umma_commit(bars->upd_full + (v & 1));
      }
    }
    if (!ok) atomicExch(js.status, ST_WAIT_TIMEOUT);
    umma_commit(&bars->drain);
    for (uint32_t n = 0; n < MOE_WAIT_LIMIT; ++n)
      if (mbar_try_wait(&bars->drain, 0)) break;
  }

  // 32 accumulator columns of this thread's row against the 64 bytes of bf16 at the same place of a
  // box: f(old, accumulator) -> new
  template <bool READ, typename F>
  static __device__ __forceinline__ void convert32(uint32_t taddr, uint32_t box, int row, int half,
                                                   F f) {
    float v[32];
    tmem_ld32(taddr, v);
    tmem_ld_wait();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t at = box + uint32_t(row) * 128u + (uint32_t((half * 4 + q) ^ (row & 7)) << 4);
      float o[8] = {};
      if constexpr (READ) {
        uint4 w;
        ld_shared_v4(at, w.x, w.y, w.z, w.w);
        unpack8(w, o);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = f(o[k], v[8 * q + k]);
      const uint4 r = pack8(o);
      st_shared_v4(at, r.x, r.y, r.z, r.w);
    }
  }

  static __device__ void converts(const NsJob& job, const NsJobs& js, int group, uint32_t tiles,
                                  uint32_t poly, uint32_t tmem, NsBars* bars) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // a quadrant's four warps: side 0 / 1 of every pair of boxes, half 0 / 1 of a box's columns
    const int quad = warp & 3, side = ((warp - 2) >> 2) & 1, half = (warp - 2) >> 3;
    const int row = quad * 32 + lane;
    const uint32_t lanes = tmem + (uint32_t(quad * 32) << 16);
    const int nt = (job.length + 127) / 128;
    float ss = 0.f;
    for (int k = 0; k < job.parts; ++k) ss += __ldcg(job.sumsq + int64_t(group) * job.parts + k);
    const float inv = 1.f / (sqrtf(ss) + js.eps);
    uint32_t loads = 0;
    // (nobody leaves after a wait that gave up: the loads from TMEM and the arrives below take all lanes of
    // a warp. With the status flagged the other waits give up soon, too, and the host sees it.)
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (!mbar_wait(bar, parity, js.status)) atomicExch(js.status, ST_WAIT_TIMEOUT);
    };
    auto arrive = [&](uint64_t* bar) {
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    for (int i = 0; i < js.steps; ++i) {
      // the parity bits of loads during the Gram pass
      for (int t = 0; t < nt; ++t)
        if (i == 0 || t >= SLOTS) loads ^= 1u << (t % SLOTS);
      const float s = i == 0 ? inv : 1.f, s2 = s * s;
      wait(&bars->acc_full, 0);
      tc_fence_after();
      if (!(s2 > 0.f))   // a norm that overflows: the direction is zero, its products may be infinite
#pragma unroll 1
        for (int c = 4 * half; c < 8 * BLOCKS; c += (c & 3) == 3 ? 5 : 1)
          st_shared_v4(poly + uint32_t(2 * (c >> 3) + side) * NS_BOX + uint32_t(row) * 128u + (c & 7) * 16,
                       0u, 0u, 0u, 0u);
#pragma unroll 1
      for (int c = s2 > 0.f ? half : 2 * BLOCKS; c < 2 * BLOCKS; c += 2)
        convert32<false>(lanes + uint32_t(c >> 1) * 128u + uint32_t(side) * 64u + uint32_t(c & 1) * 32u,
                         poly + uint32_t((c & ~1) + side) * NS_BOX, row, c & 1,
                         [&](float, float g) { return s2 * g; });
      arrive(&bars->conv_done);
      wait(&bars->acc_full, 1);
      tc_fence_after();
#pragma unroll 1
      for (int c = half; c < 2 * BLOCKS; c += 2)
        convert32<true>(lanes + uint32_t(c >> 1) * 128u + uint32_t(side) * 64u + uint32_t(c & 1) * 32u,
                        poly + uint32_t((c & ~1) + side) * NS_BOX, row, c & 1,
                        [&](float g, float g2) { return js.b * g + js.c * g2; });
      arrive(&bars->conv_done);
      for (int j = 0; j < nt; ++j) {
        const int t = nt - 1 - j, v = i * nt + j, sl = t % SLOTS;
        if (j >= SLOTS) loads ^= 1u << sl;
        wait(bars->upd_full + (v & 1), uint32_t(v >> 1) & 1u);
        wait(bars->full + sl, (loads >> sl & 1u) ^ 1u);
        tc_fence_after();
        const int live = min(128, job.length - 128 * t);
        const uint32_t d = lanes + uint32_t(v & 1) * UPD_COLS;
        const uint32_t x = tiles + uint32_t(sl) * TILE_BYTES;
        if (!TALL || quad * 32 < live) {
#pragma unroll 1
          for (int c = half; c < BOXES; c += 2) {
            const int box = (c & ~1) + side;
            if (!TALL && box * 64 + (c & 1) * 32 >= live) continue;
            convert32<true>(d + uint32_t(box) * 64u + uint32_t(c & 1) * 32u,
                            x + uint32_t(box) * NS_BOX, row, c & 1,
                            [&](float o, float u) { return s * (js.a * o + u); });
          }
        }
        arrive(bars->upd_done + (v & 1));
      }
    }
  }
};

__global__ void __launch_bounds__(NS_THREADS, 1)
    newton_schulz_kernel(const __grid_constant__ NsJobs js) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  NsBars* bars = reinterpret_cast<NsBars*>(smem + NS_DATA_BYTES);
  const int warp = threadIdx.x >> 5;
  int k = 0;
  while (k + 1 < js.n && js.job[k + 1].first_block <= int(blockIdx.x)) ++k;
  const NsJob& job = js.job[k];
  const int group = int(blockIdx.x) - job.first_block;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&job.map);
    for (int s = 0; s < NS_MAX_SLOTS; ++s) {
      mbar_init(bars->full + s, 1);
      mbar_init(bars->gram_read + s, 1);
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->conv_done, NS_EPI_WARPS);
    for (int b = 0; b < 2; ++b) {
      mbar_init(bars->upd_full + b, 1);
      mbar_init(bars->upd_done + b, NS_EPI_WARPS);
    }
    mbar_init(&bars->drain, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem, 512);
    tmem_relinquish();
    pdl_trigger();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem = bars->tmem;
  const uint32_t base = smem_u32(smem);
  if (warp == 0) {
    if (elect_one()) {
      if (job.tall) Ns<true>::copies(job, js, group, smem, bars);
      else Ns<false>::copies(job, js, group, smem, bars);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      if (job.tall) Ns<true>::mmas(job, js, base, base + NS_POLY_OFFSET_TALL, tmem, bars);
      else Ns<false>::mmas(job, js, base, base + NS_POLY_OFFSET_WIDE, tmem, bars);
    }
  } else {
    if (job.tall) Ns<true>::converts(job, js, group, base, base + NS_POLY_OFFSET_TALL, tmem, bars);
    else Ns<false>::converts(job, js, group, base, base + NS_POLY_OFFSET_WIDE, tmem, bars);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

static bool aligned16m(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
static size_t up256(size_t n) { return (n + 255) / 256 * 256; }
// blocks per matrix of the element-wise passes: four 16-byte pieces per thread
static int muon_parts(int64_t per_group) {
  return int(std::min<int64_t>(MU_PARTS, std::max<int64_t>(1, per_group / (8 * 4 * MU_THREADS))));
}

}  // namespace moe

using namespace moe;

extern "C" {

int moe_b200_muon_supported(int32_t rows, int32_t cols) {
  return (rows == 128 && cols >= 128 && cols % 32 == 0 && cols <= (1 << 20)) ||
         (cols == 256 && rows >= 256 && rows % 32 == 0 && rows <= (1 << 20));
}

size_t moe_b200_muon_scratch_bytes(const moe_b200_muon_param* params, int32_t n) {
  if (!params || n < 1) return 0;
  size_t total = 0, blocks = 0;
  for (int32_t i = 0; i < n; ++i) {
    const int64_t per = int64_t(params[i].rows) * params[i].cols;
    const size_t matrices = size_t(std::max(params[i].groups, 0));
    total += up256(matrices * size_t(per) * 2) + up256(matrices * muon_parts(per) * 4);
    blocks += matrices * muon_parts(per);
  }
  return total + blocks * 8 + 256 * size_t((n + MU_MAX - 1) / MU_MAX);
}

int moe_b200_muon_step(const moe_b200_muon_param* params, int32_t n, float grad_weight,
                       float momentum, float decay, int32_t steps, float a, float b, float c,
                       float eps, float* norms, void* scratch, size_t scratch_bytes,
                       int32_t* n_launches, int32_t* status, void* stream) {
  if (n < 1 || steps < 1) return MOE_B200_ERR_SHAPE;
  if (!params || !norms || !scratch || !status) return MOE_B200_ERR_NULL;
  if (scratch_bytes < moe_b200_muon_scratch_bytes(params, n)) return MOE_B200_ERR_SCRATCH;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  for (int32_t i = 0; i < n; ++i) {
    const moe_b200_muon_param& q = params[i];
    if (!moe_b200_muon_supported(q.rows, q.cols)) return MOE_B200_ERR_UNSUPPORTED;
    if (q.groups < 1 || q.groups > 65535) return MOE_B200_ERR_SHAPE;
    if (!q.p || !q.grad || !q.buf) return MOE_B200_ERR_NULL;
    if (!aligned16m(q.p) || !aligned16m(q.grad) || !aligned16m(q.buf)) return MOE_B200_ERR_ALIGN;
  }
  if (cudaFuncSetAttribute(newton_schulz_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           NS_SMEM) != cudaSuccess)
    return MOE_B200_ERR_CUDA;
  // a tall matrix takes about three times as long as a wide one: first in the grid
  std::vector<int32_t> order(n);
  for (int32_t i = 0; i < n; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
    return int64_t(params[x].rows) * params[x].cols * (params[x].cols == 256 && params[x].rows != 128 ? 2 : 1) >
           int64_t(params[y].rows) * params[y].cols * (params[y].cols == 256 && params[y].rows != 128 ? 2 : 1);
  });
  char* at = static_cast<char*>(scratch);
  int launched = 0;
  for (int32_t i0 = 0; i0 < n; i0 += MU_MAX) {
    MuonTensors ts{};
    NsJobs js{};
    ts.n = js.n = std::min(MU_MAX, n - i0);
    js.steps = steps;
    js.a = a;
    js.b = b;
    js.c = c;
    js.eps = eps;
    js.status = status;
    int64_t blocks = 0;
    int32_t matrices = 0;
    for (int k = 0; k < ts.n; ++k) {
      const moe_b200_muon_param& q = params[order[i0 + k]];
      const int64_t per = int64_t(q.rows) * q.cols;
      MuonTensor& t = ts.t[k];
      t.grad = static_cast<const uint4*>(q.grad);
      t.buf = static_cast<uint4*>(q.buf);
      t.p = q.p;
      t.p_is_fp32 = q.p_is_fp32;
      t.groups = q.groups;
      t.parts = muon_parts(per);
      t.pieces = int32_t(per / 8);
      t.step = q.step;
      t.first_block = blocks;
      blocks += int64_t(t.groups) * t.parts;
      t.dir = reinterpret_cast<uint4*>(at);
      at += up256(size_t(q.groups) * size_t(per) * 2);
      t.sumsq = reinterpret_cast<float*>(at);
      at += up256(size_t(q.groups) * t.parts * 4);
      NsJob& j = js.job[k];
      j.sumsq = t.sumsq;
      j.parts = t.parts;
      j.tall = q.rows != 128;
      j.length = j.tall ? q.rows : q.cols;
      j.first_block = matrices;
      matrices += q.groups;
      const uint64_t dims[3] = {uint64_t(q.cols), uint64_t(q.rows), uint64_t(q.groups)};
      const uint64_t strides[2] = {uint64_t(q.cols) * 2, uint64_t(per) * 2};
      const uint32_t box[3] = {64, 128, 1};
      if (!make_map(&j.map, t.dir, 3, dims, strides, box)) return MOE_B200_ERR_CUDA;
    }
    if (blocks > (int64_t(1) << 30)) return MOE_B200_ERR_SHAPE;
    launch_pdl(muon_direction_kernel, dim3(unsigned(blocks)), dim3(MU_THREADS), 0, st, ts,
               grad_weight, momentum, i0 == 0 ? norms : nullptr);
    launch_pdl(newton_schulz_kernel, dim3(unsigned(matrices)), dim3(NS_THREADS), size_t(NS_SMEM), st,
               js);
    float* partials = reinterpret_cast<float*>(at);
    at += up256(size_t(blocks) * 8);
    launch_pdl(muon_apply_kernel, dim3(unsigned(blocks)), dim3(MU_THREADS), 0, st, ts, decay,
               partials, norms);
    launched += 3;
    if (cudaGetLastError() != cudaSuccess) return MOE_B200_ERR_CUDA;
  }
  if (n_launches) *n_launches = launched;
  return MOE_B200_OK;
}

}  // extern "C"
