// Definition of launch_hist_grid<P>; included only by the per-plugin
// translation units that instantiate it.
#pragma once

#include "pd_hist_grid.cuh"
#include "pd_rtc.cuh"

namespace pd {

template <class P, uint32_t TP, int SPI>
static int launch_hist_grid_as(pd_ctx *ctx, const HistGrid &g) {
  using FeatT = typename P::feat_t;
  auto kern = k_hist<P, TP, SPI>;
  PD_TRY(allow_smem(ctx, kern, g.smem));
  // carve out only the shared memory the resident CTAs need; the rest stays L1
  // for the probe gathers (resident CTAs are register-limited; search form: 3 at 2
  // samples per iteration, 2 at 4 or 8)
  const int resident = TP == 0 ? kRankCtas : SPI <= 2 ? 3 : 2;
  cudaFuncAttributes fa;
  PD_CUDA(cudaFuncGetAttributes(&fa, kern));
  const size_t per_cta = g.smem + fa.sharedSizeBytes + 1024;  // dynamic + static + reserved
  const int pct = (int)std::min<size_t>(100, (resident * per_cta * 100 + 233471) / 233472);
  PD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
  if (g.queue) PD_CUDA(cudaMemsetAsync(g.queue, 0, 4, ctx->stream));
  // Without a queue the grid is the work list and the hardware scheduler keeps
  // every SM full; with one, resident CTAs pull the tiles in list order.
  const uint64_t most = 0x7fffffffull / g.tiles;  // items of one grid
  for (uint64_t b = 0; b < g.n_items; b += most) {
    const uint64_t cnt = std::min<uint64_t>(g.n_items - b, most);
    const unsigned grid = g.queue ? (unsigned)std::min<uint64_t>(cnt * g.tiles, (uint64_t)ctx->n_sms * resident)
                                  : (unsigned)(cnt * g.tiles);
    kern<<<grid, hist_threads(TP), g.smem, ctx->stream>>>(
        g.ds, g.rec, g.items + b, (uint32_t)cnt, g.queue, static_cast<const FeatT *>(g.cand_feat),
        static_cast<const FeatT *>(g.cand_thr), g.hist, g.F, g.T, g.K, g.fs, g.thr_lo, g.thr_span);
    PD_CUDA(cudaGetLastError());
    ctx->launches++;
    if (g.queue) break;  // a persistent list holds fewer than 2^31 tiles
  }
  return PD_OK;
}

// The small nodes of one class bucket: k_hist_small<P, NC>, one CTA per tile.
template <class P, int NC>
static int launch_small_as(pd_ctx *ctx, const HistGrid &g, const WorkItem *items, uint64_t n, size_t smem,
                           cudaStream_t st) {
  using FeatT = typename P::feat_t;
  auto kern = k_hist_small<P, NC>;
  PD_TRY(allow_smem(ctx, kern, smem));
  PD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, small_carveout(NC, smem)));
  const uint64_t most = 0x7fffffffull / g.tiles;
  for (uint64_t b = 0; b < n; b += most) {
    const uint64_t cnt = std::min<uint64_t>(n - b, most);
    kern<<<(unsigned)(cnt * g.tiles), small_threads(NC), smem, st>>>(
        g.ds, g.rec, items + b, static_cast<const FeatT *>(g.cand_feat), static_cast<const FeatT *>(g.cand_thr), g.F,
        g.T, g.K, g.fs, g.thr_lo, g.thr_span);
    PD_CUDA(cudaGetLastError());
    ctx->launches++;
  }
  return PD_OK;
}

template <class P>
static int launch_small(pd_ctx *ctx, const HistGrid &g) {
  const WorkItem *items = g.items + g.n_items;
  for (int b = 0; b < 4; b++) {
    const auto &s = g.small[b];
    if (!s.n_items) continue;
    cudaStream_t st;
    PD_TRY(hist_stream(ctx, g, b, &st));
    switch (s.nc) {
      case 4: PD_TRY((launch_small_as<P, 4>(ctx, g, items, s.n_items, s.smem, st))); break;
      case 8: PD_TRY((launch_small_as<P, 8>(ctx, g, items, s.n_items, s.smem, st))); break;
      case 16: PD_TRY((launch_small_as<P, 16>(ctx, g, items, s.n_items, s.smem, st))); break;
      case 32: PD_TRY((launch_small_as<P, 32>(ctx, g, items, s.n_items, s.smem, st))); break;
      default: return set_error(PD_ERR_STATE, "no small-node kernel of %d classes", s.nc);
    }
    PD_TRY(hist_join(ctx, b, st));
    items += s.n_items;
  }
  return PD_OK;
}

template <class P, uint32_t TP>
static int launch_hist_grid_tp(pd_ctx *ctx, const HistGrid &g) {
  switch (ctx->hist_spi) {
    case 2: return launch_hist_grid_as<P, TP, 2>(ctx, g);
    case 4: return launch_hist_grid_as<P, TP, 4>(ctx, g);
    case 8: return launch_hist_grid_as<P, TP, 8>(ctx, g);
    default: return set_error(PD_ERR_INVALID, "hist_spi %u", ctx->hist_spi);
  }
}

template <class P>
static int launch_big(pd_ctx *ctx, const HistGrid &g) {
  switch (g.TP) {
    case 0: return ctx->hist_spi == 8 ? launch_hist_grid_as<P, 0, 8>(ctx, g) : launch_hist_grid_as<P, 0, 4>(ctx, g);
    case 2: return launch_hist_grid_tp<P, 2>(ctx, g);
    case 4: return launch_hist_grid_tp<P, 4>(ctx, g);
    case 8: return launch_hist_grid_tp<P, 8>(ctx, g);
    case 16: return launch_hist_grid_tp<P, 16>(ctx, g);
    case 32: return launch_hist_grid_tp<P, 32>(ctx, g);
    case 64: return launch_hist_grid_tp<P, 64>(ctx, g);
    case 128: return launch_hist_grid_tp<P, 128>(ctx, g);
    case 256: return launch_hist_grid_tp<P, 256>(ctx, g);
    case 512: return launch_hist_grid_tp<P, 512>(ctx, g);
    default: return set_error(PD_ERR_UNSUPPORTED, "n_thresholds %u", g.T);
  }
}

template <class P>
int launch_hist_grid(pd_ctx *ctx, const HistGrid &g) {
  if (g.ev_before) PD_CUDA(cudaEventRecord(g.ev_before, ctx->stream));
  PD_TRY(hist_fork(ctx, g));
  if (g.n_items) PD_TRY(launch_big<P>(ctx, g));
  return launch_small<P>(ctx, g);
}

}  // namespace pd
