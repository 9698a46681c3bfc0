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
    int nc;               // k_hist_small<P, nc>
    bool may;             // a level of this training call may need it
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

// The launches of a grid -- k_hist, then the small-node kernels -- write different
// nodes' results and run side by side: the first on the context's stream, the others
// on side streams forked before it, each joined right behind its launch, so that the
// context's stream alone orders everything else.  One after the other, each left SMs
// idle at its end (a level of 300 640x480 maps has four, the small ones 0.1-1.5 ms with
// 20-40 % of the issue slots used).  Histogram time of a tree, one stream -> five: RGB
// features, 21 classes 23.8 -> 20.7 ms; images of three sizes, depth 20 35.0 -> 32.5;
// 640x480 depth maps 108.5 -> 105.5.  The small launches on one side stream: 22.4 and
// 33.9 for the first two, on two: 21.1 and 33.0.
inline int hist_fork(pd_ctx *ctx, const HistGrid &g) {
  int n = g.n_items != 0;
  for (const auto &s : g.small) n += s.n_items != 0;
  if (n > 1) PD_CUDA(cudaEventRecord(ctx->hist_fork, ctx->stream));
  return PD_OK;
}
// The stream of small launch b.
inline int hist_stream(pd_ctx *ctx, const HistGrid &g, int b, cudaStream_t *st) {
  bool first = g.n_items == 0;
  for (int i = 0; i < b; i++) first &= g.small[i].n_items == 0;
  *st = first ? ctx->stream : ctx->hist_side[b];
  if (!first) PD_CUDA(cudaStreamWaitEvent(*st, ctx->hist_fork, 0));
  return PD_OK;
}
inline int hist_join(pd_ctx *ctx, int b, cudaStream_t st) {
  if (st == ctx->stream) return PD_OK;
  PD_CUDA(cudaEventRecord(ctx->hist_join[b], st));
  PD_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->hist_join[b], 0));
  return PD_OK;
}

template <class P>
int launch_hist_grid(pd_ctx *ctx, const HistGrid &g);
// The run-time compiled histogram kernel of a user feature (pd_rtc.cu).
int launch_hist_grid_rtc(pd_ctx *ctx, const HistGrid &g);

extern template int launch_hist_grid<DepthDiff2>(pd_ctx *, const HistGrid &);
extern template int launch_hist_grid<DepthDiff1>(pd_ctx *, const HistGrid &);
extern template int launch_hist_grid<ChannelDiff>(pd_ctx *, const HistGrid &);

}  // namespace pd
