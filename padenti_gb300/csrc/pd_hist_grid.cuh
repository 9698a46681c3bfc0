// Launch of the histogram kernel over a work list.  The kernel has one
// instantiation per (plugin, padded threshold rows, samples per iteration); each
// plugin's set is compiled in its own translation unit (pd_hist_<plugin>.cu) so
// that the build compiles them in parallel.
#pragma once

#include <algorithm>

#include "pd_ctx.cuh"
#include "pd_train_kernels.cuh"

namespace pd {

struct HistGrid {
  DevSet ds;
  const SampleRec *rec;   // active samples of the work list's ranges
  const WorkItem *items;  // device work list: the items of k_hist, then of each small launch
  uint64_t n_items;       // items of k_hist (tiles CTAs each)
  uint32_t tiles;
  // rank-table form: small nodes (fused split) by the class rows of their kernel
  struct Small {
    int nc;               // k_hist_small<P, nc>; 0: no such launch
    uint64_t n_items;
    size_t smem;
  } small[4];
  const void *cand_feat, *cand_thr;
  uint32_t *hist;
  uint32_t F, T, K, TP;   // TP = threshold rows padded to a power of two above T; 0: rank-table form
  int32_t thr_lo;         // rank-table form: the thresholds lie in [thr_lo, thr_lo + thr_span]
  uint32_t thr_span;
  size_t smem;            // dynamic shared memory per CTA
  FusedSplit fs;
  cudaEvent_t ev_before;  // recorded just before the first launch (may be null)
  unsigned *queue;        // persistent launch: the work counter (zeroed here), null: one CTA per item
};

// Shared-memory carve-out (per cent of 228 KB) for the resident CTAs of a
// k_hist_small<., NC> launch; the rest stays L1.
inline int small_carveout(int NC, size_t smem) {
  const size_t all = (size_t)small_ctas(NC) * (smem + 1024 + 1024);
  return (int)std::min<size_t>(100, (all * 100 + 233471) / 233472);
}

template <class P>
int launch_hist_grid(pd_ctx *ctx, const HistGrid &g);
// The run-time compiled histogram kernel of a user feature (pd_rtc.cu).
int launch_hist_grid_rtc(pd_ctx *ctx, const HistGrid &g);

extern template int launch_hist_grid<DepthDiff2>(pd_ctx *, const HistGrid &);
extern template int launch_hist_grid<DepthDiff1>(pd_ctx *, const HistGrid &);
extern template int launch_hist_grid<ChannelDiff>(pd_ctx *, const HistGrid &);

}  // namespace pd
