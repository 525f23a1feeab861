// The weight gradients' split-K work items: how many a run has, the rows of each, and the order they are
// walked in. (No CUDA in here: the tests compile it for the host too.)
#pragma once

#ifdef __CUDACC__
#define MOE_ORDER_FN __host__ __device__ __forceinline__
#else
#define MOE_ORDER_FN inline
#endif

namespace moe {

constexpr int WGRAD_BK = 64;   // rows of a K block

// Number of work items of a run of `rows` rows.
MOE_ORDER_FN int wgrad_chunks(int rows, int ks_rows) {
  return rows <= ks_rows ? 1 : (rows + ks_rows - 1) / ks_rows;
}

struct WgradRuns {
  const int* start;   // routed: [n_groups + 1], run g ends where run g + 1 starts; fixed: zeros
  int fixed_rows;     // fixed: every run has rows [0, fixed_rows); -1: routed
  MOE_ORDER_FN int end(int g) const { return fixed_rows >= 0 ? fixed_rows : start[g + 1]; }
};
struct WgradRows {
  int row0, blocks;   // K blocks from row0 on (0: the only item of an empty run)
};
// Item `chunk` of run g.
MOE_ORDER_FN WgradRows wgrad_rows(const WgradRuns& r, int ks_rows, int g, int chunk) {
  WgradRows w;
  w.row0 = r.start[g] + chunk * ks_rows;
  const int left = r.end(g) - w.row0, rows = left < 0 ? 0 : left > ks_rows ? ks_rows : left;
  w.blocks = (rows + WGRAD_BK - 1) / WGRAD_BK;
  return w;
}

// Whether item k is walked before item i, by their K blocks: decreasing, ties by index. The list is read four
// items at a time; what stands behind its end has WGRAD_NO_ITEM blocks and comes before nothing.
constexpr int WGRAD_NO_ITEM = -1;
MOE_ORDER_FN bool wgrad_before(int blocks_k, int k, int blocks_i, int i) {
  return blocks_k > blocks_i || (blocks_k == blocks_i && k < i);
}

}  // namespace moe
