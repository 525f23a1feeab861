// What the decode stack (stack.cu) runs on: its sizes, its shared memory, and which shapes and devices it
// takes. (No CUDA in here: the tests compile it for the host too.)
#pragma once
#include <stdint.h>

#include <algorithm>

#include "per_device.cuh"

#ifdef __CUDACC__
#define MOE_STACK_FN __host__ __device__ inline
#else
#define MOE_STACK_FN inline
#endif

namespace moe {

constexpr int ST_H = 128;                  // hidden units per expert
constexpr int ST_SLICE = 32;               // of them in one work item
constexpr int ST_SLICES = ST_H / ST_SLICE;
constexpr int ST_STAGE = 8192;             // ring stage: [gate | up][64 d][32 units] or [2][32 units][64 d]
constexpr int ST_HALF = ST_STAGE / 2;
// 16 compute warps: the phases are chains of dependent instructions, so what counts is how few of them a
// warp has. One more warp issues the TMA loads: a box of 64-byte rows occupies the TMA unit for some
// 200 cycles, and whoever issues a part's loads stands in that queue for a microsecond. (It leaves a
// thread 96 registers; a spill would cost more, it finds no room in the L1 beside the shared memory.)
constexpr int ST_WARPS = 16;
constexpr int ST_CT = ST_WARPS * 32;       // compute threads
constexpr int ST_THREADS = ST_CT + 32;
constexpr int ST_PASS = 16;                // tokens per pass over an item (two mma column tiles)
constexpr int ST_ACC_LD = 68;              // floats between tokens of the up accumulators
constexpr int ST_ACC_BYTES = 4 * ST_PASS * ST_ACC_LD * 4;
constexpr int ST_HID_LD = 40;              // bf16 between tokens of the hidden rows (80 B: no conflicts)
constexpr int ST_MAX_T = 256;
constexpr int ST_MAX_ITEMS = 8;            // items of one CTA and layer
constexpr int ST_MAX_STAGES = 24;
constexpr int ST_PARTS = 32;               // barriers for the two parts of an item; more than stages
constexpr int ST_MAX_SLOTS = 4;            // tokens of one CTA
constexpr int ST_RED_BYTES = 16 * ST_CT;   // token phase: partial sums, then the router's
static_assert(ST_RED_BYTES <= ST_ACC_BYTES, "they share the accumulators' place");
// Router weight chunks (four columns of a row; a thread has 23 at 76 experts and d_model 576): the
// first ST_ROUTER_PRE are held in registers across the hand-over, the next are copied to the row
// buffer and the accumulators, which are free then, and ST_ROUTER_EXTRA bytes beside them, and
// ST_ROUTER_LATE more are fetched when the partial rows are in. Chunks loaded at their use cost an L2
// latency a batch.
constexpr int ST_ROUTER_PRE = 5, ST_ROUTER_LATE = 10, ST_ROUTER_EXTRA = 8192;
static_assert(ST_PASS == ST_WARPS, "a warp has one token of a pass");
static_assert(ST_MAX_ITEMS <= ST_WARPS, "a warp lists one item's tokens");
constexpr int ST_MAX_GROUPS = 256;         // routed and shared experts
constexpr int ST_MAX_SMEM = 232448;        // shared memory of a block

// Shared memory behind the ring, in order.
struct StackSmem {
  int xs, acc, hid, list, xrow, res, tokw, lg, bars, misc, total;
};
MOE_STACK_FN StackSmem stack_smem(int T, int D, int n_stages, int extra) {
  const int dpad = (D + 63) / 64 * 64;
  StackSmem s;
  int at = n_stages * ST_STAGE;
  auto take = [&](int bytes) {
    const int r = at;
    at += (bytes + 15) / 16 * 16;
    return r;
  };
  take(extra);                                         // router weight chunks, with xs and acc
  s.xs = take(ST_PASS * (dpad * 2 + 16));              // token rows of a pass
  s.acc = take(ST_ACC_BYTES);                          // up accumulators; token phase: partial sums
  s.hid = take((T + ST_PASS - 1) / ST_PASS * ST_PASS * ST_HID_LD * 2);
  s.list = take(2 * ST_MAX_ITEMS * T * 2);             // an item's tokens, and their pairs
  s.xrow = take(dpad * 4);                             // token phase: the row, fp32
  s.res = take(ST_MAX_SLOTS * D * 2);                  // residual rows of this CTA's tokens
  s.tokw = take(ST_MAX_SLOTS * 16 * 4);                // their pairs' weights
  s.lg = take(2 * ST_MAX_GROUPS * 4);                  // logits, their sort keys
  s.bars = take(2 * ST_PARTS * 8);
  s.misc = take(16 + ST_MAX_ITEMS * 4 + ST_MAX_ITEMS * 16);   // flags, token counts, items
  s.total = at;
  return s;
}

// What the grid needs to know of a device. Its CTAs wait on one another, so that all of them have to be
// resident: one per SM that this process has, which may be a part of the device.
struct StackDevice {
  int sms = 0, blocks_per_sm = 0;
  bool cooperative = false;
  int grid() const { return cooperative && blocks_per_sm > 0 ? sms : 0; }   // 0: cannot be launched
};

// The shape side of a launch; false: the layer-by-layer path is the one that takes it.
struct StackShape {
  int sh_tokens, sh_blocks, n_items, n_stages, router_extra, smem;
};
inline bool stack_shape(const StackDevice& dev, int64_t T, int D, int H, int E, int S, int k, StackShape* o) {
  if (T < 1 || T > ST_MAX_T || H != ST_H || D < 64 || D % 32 != 0 || D > 1024 || E < 4 ||
      E % 4 != 0 || S < 0 || E + S > ST_MAX_GROUPS || k < 1 || k > E || k + S > 16)
    return false;
  const int grid = dev.grid();
  if (T > int64_t(ST_MAX_SLOTS) * grid) return false;
  // a shared expert sees every token: one pass's worth of them per work item keeps it in the range of
  // the others, as long as that does not give every CTA more items
  o->sh_tokens = int(std::min<int64_t>(T, T > 128 ? 2 * ST_PASS : ST_PASS));
  o->sh_blocks = int((T + o->sh_tokens - 1) / o->sh_tokens);
  o->n_items = ST_SLICES * (E + S * o->sh_blocks);
  if (o->n_items > ST_MAX_ITEMS * grid) return false;
  const int limit = ST_MAX_SMEM - 1024, n_in = (D + 63) / 64;
  for (int extra : {ST_ROUTER_EXTRA, 0}) {
    const int rest = stack_smem(int(T), D, 0, extra).total;
    o->router_extra = extra;
    o->n_stages = std::min((limit - rest) / ST_STAGE, ST_MAX_STAGES);
    if (limit > rest && o->n_stages >= n_in) break;   // an item's up weights are there at once
  }
  if (o->n_stages < n_in) return false;
  o->smem = stack_smem(int(T), D, o->n_stages, o->router_extra).total + 1024;
  return true;
}

}  // namespace moe
