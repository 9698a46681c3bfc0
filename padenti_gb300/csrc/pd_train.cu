// Host orchestration of the training pass: CLTreeTrainer::train
// (cl_tree_trainer_impl.hpp:203-255) re-designed for one GPU with the whole
// training set resident in HBM.  Per depth: candidate table, histogram work
// list over all frontier nodes (one launch per histogram slice), best split on
// the device, finalize on the host (it is O(frontier)), device tree update,
// reassignment and stable regrouping of the active samples.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <vector>

#include "pd_ctx.cuh"
#include "pd_hist_grid.cuh"
#include "pd_rtc.cuh"
#include "pd_predict_kernels.cuh"
#include "pd_train_kernels.cuh"

namespace pd {

// Threshold rows padded to the next power of two above T, so the branch-free
// search needs no bounds test.
static uint32_t padded_rows(uint32_t T) {
  uint32_t p = 1;
  while (p < T + 1) p <<= 1;
  return p;
}

// Shared memory of a histogram launch: packed tile histogram, threshold table
// and, when the launch has fused-split items, the larger of the table and the
// fused scratch (gains + packed left totals) that overlays it.
static size_t hist_smem(const pd_ctx *ctx, uint32_t T, bool fused = true) {
  const size_t hist = (size_t)ctx->cfg.n_classes * (T + 1) * 32 * 4;  // rank T rows are never read
  const size_t thr = (size_t)padded_rows(T) * kTileF * feat_size(ctx->cfg.feat_type);
  const size_t scratch = (size_t)T * kTileF * 4 + (size_t)T * 32 * 4;
  return hist + (fused ? std::max(thr, scratch) : thr);
}

// Shared memory of a CTA of the rank-table form with `rows` class rows and
// `threads` threads: packed tile histogram, `first` bits, table, staged words.
static size_t rank_smem(uint32_t rows, uint32_t T, uint32_t span, int threads) {
  return (size_t)rows * (T + 1) * 32 * 4 + (size_t)kTileF * ((T + 31) / 32) * 4 + (size_t)rank_words(span) * 64 * 4 +
         (size_t)threads / 32 * 64 * 16;
}
constexpr size_t kRankSmemMax = 227 * 1024 - 4096;  // dynamic; the kernels' static arrays take less than 4 KB

// Whether the histogram kernels take the rank-table form: the thresholds are the
// draws of [thr_low, thr_up] without wrapping, the table has at most
// kRankWordsMax words a column, and a CTA's histogram of all classes fits the
// shared memory beside it (the search form takes what is left, such as 64 classes
// with many thresholds).  The widest table still pays at every threshold count:
// histogram time of a tree (100 maps of 640x480, 1000 candidates, depth 13, 3 classes),
// search / table: thresholds in +-1020, 1 of them 9.1 / 7.4 ms, 4 10.0 / 7.8, 50 13.2 /
// 10.8; in +-500, 1 9.0 / 6.8, 50 13.2 / 8.0.
bool rank_form(const pd_ctx *ctx, const pd_train_params *p, const PropSrc *prop) {
  if (prop) {  // proposals are clamped to the network's bounds: they must be these
    const int D = ctx->cfg.feat_dim;
    if (prop->lo[D] != (float)p->thr_low || prop->span[D] != (float)((int64_t)p->thr_up - p->thr_low) ||
        p->thr_low < -(1 << 23) || p->thr_up > (1 << 23))
      return false;
  }
  const int64_t lo = p->thr_low, hi = p->thr_up, span = hi - lo;
  const int64_t fmax = ctx->cfg.feat_type == PD_FEAT_I16 ? 32767 : (1 << 29);
  if (span < 0 || lo < -fmax || hi > fmax || span + 1 >= (int64_t)kRankWordsMax * 16) return false;
  return rank_smem((uint32_t)ctx->cfg.n_classes, p->n_thresholds, (uint32_t)span, kRankThreads) <= kRankSmemMax;
}

// The class rows of the small-node kernel for a node with nc classes present (an
// index into kSmallRows), or -1 when none fits.  A user feature's kernels are
// compiled on first use: only two of them.
constexpr int kSmallRows[4] = {4, 8, 16, 32};
static int small_bucket(const pd_ctx *ctx, const pd_train_params *p, uint32_t nc) {
  const uint32_t span = (uint32_t)(p->thr_up - p->thr_low);
  for (int b = is_user_plugin(ctx) ? 1 : 0; b < 4; b++) {
    if (is_user_plugin(ctx) && b == 2) continue;
    if ((int)nc <= kSmallRows[b])
      return rank_smem(kSmallRows[b], p->n_thresholds, span, small_threads(kSmallRows[b])) <= kRankSmemMax ? b : -1;
  }
  return -1;
}

static DevSet devset(const pd_ctx *ctx) {
  DevSet d;
  d.magic = ctx->magic_tab.as<uint32_t>();
  d.pixels = ctx->pixels.as<uint8_t>();
  d.img_off = ctx->img_off.as<uint64_t>();
  d.img_wh = ctx->img_wh.as<uint32_t>();
  d.s_xy = ctx->s_xy.as<uint32_t>();
  d.s_img = ctx->s_img.as<uint32_t>();
  d.s_label = ctx->s_label.as<uint8_t>();
  const bool tf = ctx->tree_feature && ctx->nm_pixels;
  d.nodes = tf ? ctx->nm_map[ctx->nm_cur].as<int32_t>() : nullptr;
  d.map_off = tf ? ctx->nm_off.as<uint64_t>() : nullptr;
  d.tree_lc = ctx->t_lc.as<int32_t>();
  d.tree_post = ctx->t_post.as<float>();
  d.n_classes = (uint32_t)ctx->cfg.n_classes;
  d.tree_level = ctx->nm_level;
  d.tree_nodes = ctx->nm_nodes;
  return d;
}

int ensure_log2_table(pd_ctx *ctx, uint64_t n) {
  if (n <= ctx->log2_len) return PD_OK;
  PD_CHECK(n <= (1ull << 32), PD_ERR_UNSUPPORTED, "log2 table of %llu entries", (unsigned long long)n);
  PD_TRY(ctx->log2_tab.ensure(n * sizeof(double)));
  const DD inv = dd_inv_ln2();
  k_log2_table<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(ctx->log2_tab.as<double>(), n, inv);
  PD_CUDA(cudaGetLastError());
  const uint32_t m = (uint32_t)std::min<uint64_t>(n, kXlog2Len);
  PD_TRY(ctx->xlog2_tab.ensure((size_t)kXlog2Len * sizeof(float)));
  k_xlog2_table<<<(m + 255) / 256, 256, 0, ctx->stream>>>(ctx->xlog2_tab.as<float>(), ctx->log2_tab.as<double>(), m);
  PD_CUDA(cudaGetLastError());
  ctx->log2_len = n;
  return PD_OK;
}

int map_training_pixels(pd_ctx *ctx, uint64_t bytes) {
  return dispatch_config(ctx->cfg, [&]<class P>() -> int {
    if constexpr (P::kTrainMapsZero) {
      static_assert(sizeof(typename P::img_t) == 2, "zero mapping of 16-bit images");
      const uint64_t n = is_user_plugin(ctx) ? 0 : bytes / 2;  // a user feature reads the images as given
      if (n) {
        k_zero_to_background<<<4 * 152, 256, 0, ctx->stream>>>(ctx->pixels.as<uint16_t>(), n);
        PD_CUDA(cudaGetLastError());
      }
    }
    return PD_OK;
  });
}

int build_sample_records(pd_ctx *ctx, uint64_t S) {
  PD_TRY(ctx->s_rec.ensure(S * sizeof(SampleRec) + sizeof(SampleRec)));
  if (!S) return PD_OK;
  return dispatch_config(ctx->cfg, [&]<class P>() -> int {
    const dim3 grid((unsigned)((S + 255) / 256));
    if (is_user_plugin(ctx)) {
      const RtcKernels *rk = nullptr;
      PD_TRY(rtc_kernels(ctx, &rk));
      DevSet ds = devset(ctx);
      uint32_t n = (uint32_t)S;
      SampleRec *rec = ctx->s_rec.as<SampleRec>();
      void *args[] = {&ds, &n, &rec};
      return rtc_launch(ctx, rk->build_rec, grid, dim3(256), 0, args);
    }
    if constexpr (!P::kRtcOnly) {
      k_build_rec<P><<<grid, 256, 0, ctx->stream>>>(devset(ctx), (uint32_t)S, ctx->s_rec.as<SampleRec>());
      PD_CUDA(cudaGetLastError());
    }
    return PD_OK;
  });
}

int init_tables(pd_ctx *ctx) {
  PD_TRY(ctx->magic_tab.ensure(65536 * 4));
  k_magic_table<<<256, 256, 0, ctx->stream>>>(ctx->magic_tab.as<uint32_t>());
  PD_CUDA(cudaGetLastError());
  return PD_OK;
}

static CandBounds bounds(const pd_train_params *p, int D, uint32_t f_base = 0) {
  CandBounds b;
  memset(&b, 0, sizeof(b));
  b.f_base = f_base;
  for (int d = 0; d < D; d++) {
    b.low[d] = p->feat_low[d];
    b.up[d] = p->feat_up[d];
  }
  b.thr_lo = p->thr_low;
  b.thr_hi = p->thr_up;
  return b;
}

static int check_params(const pd_ctx *ctx, const pd_train_params *p) {
  PD_CHECK(p, PD_ERR_INVALID, "null params");
  PD_CHECK(p->n_features >= 1 && p->n_thresholds >= 1, PD_ERR_INVALID, "n_features and n_thresholds must be >= 1");
  PD_CHECK(p->n_thresholds <= PD_MAX_THRESHOLDS, PD_ERR_UNSUPPORTED, "n_thresholds %u > %d",
           p->n_thresholds, PD_MAX_THRESHOLDS);
  const size_t smem = hist_smem(ctx, p->n_thresholds);
  PD_CHECK(smem <= 227 * 1024, PD_ERR_UNSUPPORTED,
           "nClasses*nThresholds too large for one shared-memory histogram tile (%zu bytes)", smem);
  return PD_OK;
}

// Lays the results of a slice of n nodes out in one buffer (kept; grown as needed).
static int set_results(pd_ctx *ctx, uint32_t n) {
  auto up = [](size_t v) { return (v + 15) / 16 * 16; };
  const size_t K = ctx->cfg.n_classes, par = up((size_t)n * (ctx->cfg.feat_dim + 1) * feat_size(ctx->cfg.feat_type));
  const size_t out = up((size_t)n * sizeof(SplitOut)), cl = up((size_t)n * K * 4);
  PD_TRY(ctx->split_res.ensure(out + cl + par + 16));  // 16: SplitArgs::rechecked
  uint8_t *b = ctx->split_res.as<uint8_t>();
  ctx->res_out = b;
  ctx->res_cl = reinterpret_cast<uint32_t *>(b + out);
  ctx->res_par = b + out + cl;
  ctx->res_recheck = reinterpret_cast<unsigned long long *>(b + out + cl + par);
  ctx->res_bytes = out + cl + par + 16;
  return PD_OK;
}

// Scratch sized for `slots` frontier nodes.
static int ensure_slice(pd_ctx *ctx, const pd_train_params *p, uint32_t slots) {
  const uint64_t F = p->n_features, T = p->n_thresholds, K = ctx->cfg.n_classes;
  const size_t fs = feat_size(ctx->cfg.feat_type);
  PD_TRY(ctx->cand_feat.ensure(slots * ctx->cfg.feat_dim * F * fs));
  PD_TRY(ctx->cand_thr.ensure(slots * T * F * fs));
  PD_TRY(ctx->cand_perm.ensure(slots * T * F));
  PD_TRY(ctx->cand_ord.ensure(slots * F * 4));
  PD_TRY(ctx->hist.ensure(slots * K * T * F * 4));
  PD_TRY(ctx->g32.ensure(slots * T * F * 4));
  return set_results(ctx, slots);
}

static uint64_t slot_bytes(const pd_ctx *ctx, const pd_train_params *p) {
  const uint64_t F = p->n_features, T = p->n_thresholds, K = ctx->cfg.n_classes;
  const uint64_t fs = feat_size(ctx->cfg.feat_type);
  return K * T * F * 4 + T * F * 4 + T * F * (fs + 1) + ctx->cfg.feat_dim * F * fs + F * 4;
}

// ----------------------------------------------------------- launches ----
// Candidate tables of n slots.  With `ordered` (and F <= kOrderMaxF) the
// columns of each slot are sorted by first-probe offset and *ord_out receives
// the column -> original index map; otherwise column f is candidate f and
// *ord_out is null.
template <class P>
static int launch_candidates(pd_ctx *ctx, const pd_train_params *p, uint32_t tree, const int32_t *d_nodes,
                             uint32_t n, bool ordered = false, const uint32_t **ord_out = nullptr,
                             const PropSrc *prop = nullptr, uint32_t f_base = 0) {
  using FeatT = typename P::feat_t;
  const uint32_t F = p->n_features;
  const uint64_t total = (uint64_t)n * F;
  const uint32_t *ord = nullptr;
  if (ord_out) *ord_out = nullptr;
  if (!total) return PD_OK;
  const CandBounds b = bounds(p, P::kFeatDim, f_base);
  if (ordered && F <= kOrderMaxF) {
    uint32_t N = 1;
    while (N < F) N <<= 1;
    const size_t osmem = (size_t)N * 8;
    if (is_user_plugin(ctx)) {
      const RtcKernels *rk = nullptr;
      PD_TRY(rtc_kernels(ctx, &rk));
      PD_TRY(rtc_set_smem(ctx, rk->cand_order, osmem));
      uint32_t tr = tree, f_ = F;
      CandBounds bb = b;
      uint32_t *o = ctx->cand_ord.as<uint32_t>();
      PropSrc ps = prop ? *prop : PropSrc{};
      void *args[] = {&d_nodes, &tr, &f_, &bb, &o, &ps};
      PD_TRY(rtc_launch(ctx, rk->cand_order, dim3(n), dim3(kOrderThreads), osmem, args));
    } else if constexpr (!P::kRtcOnly) {
      PD_TRY(allow_smem(ctx, k_cand_order<P>, osmem));
      k_cand_order<P><<<n, kOrderThreads, osmem, ctx->stream>>>(d_nodes, tree, F, b, ctx->cand_ord.as<uint32_t>(),
                                                                prop ? *prop : PropSrc{});
      PD_CUDA(cudaGetLastError());
      ctx->launches++;
    }
    ord = ctx->cand_ord.as<uint32_t>();
  }
  // draws lie in [lo, hi] (no narrowing wrap) and their offsets fit 24 bits:
  // value and index sort as one word
  const int64_t span = (int64_t)p->thr_up - p->thr_low;
  const bool packed = span >= 0 && span < (1 << 24) && (sizeof(FeatT) == 4 || span <= 32767);
  const unsigned grid = (unsigned)((total + kCandThreads - 1) / kCandThreads);
  const uint32_t T = p->n_thresholds;
  if (packed && T <= 64 && ctx->cand_regs) {
    // keys sorted in registers
    auto rk = T <= 16 ? k_candidates_reg<FeatT, 16> : (T <= 32 ? k_candidates_reg<FeatT, 32> : k_candidates_reg<FeatT, 64>);
    rk<<<grid, kCandThreads, (size_t)T * kCandThreads * 4, ctx->stream>>>(d_nodes, n, tree, F, T, P::kFeatDim, b, ord, ctx->cand_feat.as<FeatT>(),
                                               ctx->cand_thr.as<FeatT>(), ctx->cand_perm.as<uint8_t>(),
                                               prop ? *prop : PropSrc{});
    PD_CUDA(cudaGetLastError());
    ctx->launches++;
    if (ord_out) *ord_out = ord;
    return PD_OK;
  }
  const size_t smem = (size_t)p->n_thresholds * kCandThreads * (packed ? 4 : sizeof(FeatT) + 1);
  auto kern = packed ? k_candidates<FeatT, true> : k_candidates<FeatT, false>;
  PD_TRY(allow_smem(ctx, kern, smem));
  kern<<<grid, kCandThreads, smem, ctx->stream>>>(
      d_nodes, n, tree, F, p->n_thresholds, P::kFeatDim, b, ord, ctx->cand_feat.as<FeatT>(),
      ctx->cand_thr.as<FeatT>(), ctx->cand_perm.as<uint8_t>(), prop ? *prop : PropSrc{});
  PD_CUDA(cudaGetLastError());
  ctx->launches++;
  if (ord_out) *ord_out = ord;
  return PD_OK;
}

// Builds the work list of slots [0, n) whose samples are act[off[i], off[i+1])
// and launches the histogram kernels.  With `split_slots` non-null, nodes whose
// samples fit one work item get their split fused into the histogram kernel (multi
// = 2, rows never written) and the other slots are returned for the split kernels;
// h_class_tot: their class totals [n][K] on the host; *d_split_list: those slots on the
// device.
template <class P>
static int launch_hist(pd_ctx *ctx, const pd_train_params *p, const uint64_t *off, uint32_t n,
                       const SampleRec *d_rec, uint64_t *n_items_out, cudaEvent_t ev_before = nullptr,
                       cudaEvent_t ev_after = nullptr, std::vector<uint32_t> *split_slots = nullptr,
                       const uint32_t *d_class_tot = nullptr, const uint32_t *h_class_tot = nullptr,
                       const uint32_t *d_ord = nullptr, const PropSrc *prop = nullptr,
                       const uint32_t **d_split_list = nullptr) {
  using FeatT = typename P::feat_t;
  const uint32_t F = p->n_features, T = p->n_thresholds, K = ctx->cfg.n_classes;
  const uint32_t tiles = (F + kTileF - 1) / kTileF;
  PD_CHECK(ctx->chunk >= 1 && ctx->chunk <= kMaxChunk, PD_ERR_INVALID, "chunk %u outside [1,%u]", ctx->chunk, kMaxChunk);
  const bool rank = rank_form(ctx, p, prop);
  const uint32_t span = rank ? (uint32_t)(p->thr_up - p->thr_low) : 0u;
  // Samples per work item: the chunk, or less when the level has too few tiles to
  // fill the GPU: four items per SM, fewer when they would be small (the set-up and
  // flush of a tile cost about as much as 800 samples), one at least.  64 maps of
  // 160x120 with 200 candidates: the root's 8 CTAs of 16384 samples took 0.33 ms, its
  // 500 of 256 0.05; four items per SM on every level 0.322 ms of histograms a tree,
  // this rule 0.280.
  static constexpr uint64_t kMinChunk = 256;
  const uint64_t total = off[n] - off[0];
  const uint64_t per_sm = (total * tiles + ctx->n_sms - 1) / ctx->n_sms;
  auto round32 = [](uint64_t v) { return std::max<uint64_t>(kMinChunk, (v + 31) / 32 * 32); };
  const uint64_t items_per_sm = std::min<uint64_t>(4, std::max<uint64_t>(1, per_sm / 1024));
  const uint64_t chunk =
      rank ? std::min<uint64_t>(ctx->chunk, round32((per_sm + items_per_sm - 1) / items_per_sm)) : ctx->chunk;
  // a fused node runs on a CTA of fewer warps: on a small level only short ones do
  const uint64_t fuse_max = rank ? std::min({(uint64_t)ctx->fuse_max, chunk, round32((per_sm + 3) / 4)})
                                 : std::min<uint64_t>(ctx->fuse_max, chunk);
  // Per node: fused (a small-node launch of its class count in the rank-table form,
  // an item with multi = 2 in the search form) or chunked.  The list is written
  // straight into pinned staging: the items of k_hist -- for a persistent launch
  // largest first (by the power of two of their sample count, stable), so that the
  // last to start are the short ones -- then the small nodes by class bucket.
  const bool persist = ctx->persist;
  auto bucket = [](uint64_t cnt) { return cnt ? 63 - __builtin_clzll(cnt) : 0; };  // floor(log2), <= 15
  std::vector<int8_t> kind(n);  // -2 empty, -1 chunked, -3 fused in k_hist, b >= 0 small bucket
  uint64_t n_small[4] = {}, n_big = 0, pos[17] = {};
  for (uint32_t i = 0; i < n; i++) {
    const uint64_t cnt = off[i + 1] - off[i], chunks = (cnt + chunk - 1) / chunk;
    int k = cnt ? -1 : -2;
    if (split_slots && cnt && cnt <= fuse_max) {
      if (!rank) {
        k = -3;
      } else {
        uint32_t nc = 0;
        for (uint32_t l = 0; l < K; l++) nc += h_class_tot[(size_t)i * K + l] != 0u;
        k = small_bucket(ctx, p, nc);
      }
    }
    kind[i] = (int8_t)k;
    if (k >= 0) {
      n_small[k]++;
      continue;
    }
    n_big += chunks;
    for (uint64_t c = 0; persist && c < chunks; c++) pos[bucket(std::min<uint64_t>(cnt - c * chunk, chunk))]++;
  }
  uint64_t acc = 0;
  for (int b = 15; persist && b >= 0; b--) {  // start of each bucket, largest first
    const uint64_t c = pos[b];
    pos[b] = acc;
    acc += c;
  }
  uint64_t at[4], n_items = n_big;
  for (int b = 0; b < 4; b++) {
    at[b] = n_items;
    n_items += n_small[b];
  }
  PD_TRY(ctx->h_items.ensure(n_items * sizeof(WorkItem) + (size_t)n * 8 + 16));
  WorkItem *items = ctx->h_items.as<WorkItem>();
  uint64_t ni = 0;
  std::vector<uint32_t> zero;
  bool any_fused = false;
  for (uint32_t i = 0; i < n; i++) {
    const uint64_t b = off[i], e = off[i + 1];
    if (kind[i] == -2) {
      zero.push_back(i);
      if (split_slots) split_slots->push_back(i);
      continue;
    }
    WorkItem w;
    memset(&w, 0, sizeof(w));
    w.slot = i;
    if (kind[i] >= 0) {
      w.begin = (uint32_t)b;
      w.end = (uint32_t)e;
      w.multi = 2;
      items[at[kind[i]]++] = w;
      continue;
    }
    const uint64_t chunks = (e - b + chunk - 1) / chunk;
    if (chunks > 1) zero.push_back(i);
    any_fused |= kind[i] == -3;
    if (split_slots && kind[i] != -3) split_slots->push_back(i);
    w.multi = chunks > 1 ? 1u : (kind[i] == -3 ? 2u : 0u);
    for (uint64_t c = 0; c < chunks; c++) {
      w.begin = (uint32_t)(b + c * chunk);
      w.end = (uint32_t)std::min<uint64_t>(e, b + (c + 1) * chunk);
      items[persist ? pos[bucket(w.end - w.begin)]++ : ni] = w;
      ni++;
    }
  }
  *n_items_out = n_items * tiles;
  // one copy: the work list, the slots whose rows are added to (zeroed first), the
  // slots for the split kernels
  uint32_t *lists = reinterpret_cast<uint32_t *>(items + n_items);
  size_t n_lists = zero.size();
  if (!zero.empty()) memcpy(lists, zero.data(), zero.size() * 4);
  if (split_slots && !split_slots->empty()) {
    memcpy(lists + n_lists, split_slots->data(), split_slots->size() * 4);
    n_lists += split_slots->size();
  }
  const size_t list_bytes = n_items * sizeof(WorkItem) + n_lists * 4;
  PD_TRY(ctx->items.ensure(list_bytes + 16));
  if (list_bytes) PD_CUDA(h2d(ctx, ctx->items.ptr, items, list_bytes));
  const uint32_t *d_lists = reinterpret_cast<const uint32_t *>(ctx->items.as<WorkItem>() + n_items);
  if (d_split_list) *d_split_list = d_lists + zero.size();
  const uint64_t per_slot = (uint64_t)K * T * F;
  if (!zero.empty()) {
    k_zero_slots<<<1216, 256, 0, ctx->stream>>>(ctx->hist.as<uint32_t>(), d_lists, (uint32_t)zero.size(), per_slot);
    PD_CUDA(cudaGetLastError());
    ctx->launches++;
  }
  if (!n_items) {
    if (ev_before) PD_CUDA(cudaEventRecord(ev_before, ctx->stream));
    if (ev_after) PD_CUDA(cudaEventRecord(ev_after, ctx->stream));
    return PD_OK;
  }
  FusedSplit fs;
  memset(&fs, 0, sizeof(fs));
  if (split_slots) {
    PD_TRY(ctx->fused_scratch.ensure((size_t)n * 4 + (size_t)n * tiles * (sizeof(SplitPart) + 4 * K) + 64));
    fs.done = ctx->fused_scratch.as<unsigned>();
    fs.part_best = reinterpret_cast<SplitPart *>(ctx->fused_scratch.as<uint8_t>() + ((size_t)n * 4 + 15) / 16 * 16);
    fs.part_cl = reinterpret_cast<uint32_t *>(fs.part_best + (size_t)n * tiles);
    PD_CUDA(cudaMemsetAsync(fs.done, 0, (size_t)n * 4, ctx->stream));
    fs.class_tot = d_class_tot;
    fs.perm = ctx->cand_perm.as<uint8_t>();
    fs.L = ctx->log2_tab.as<double>();
    fs.L_len = ctx->log2_len;
    fs.xlog2 = ctx->xlog2_tab.as<float>();
    PD_TRY(ctx->parent.ensure((size_t)n * sizeof(double)));
    k_parent_term<<<(n + 127) / 128, 128, 0, ctx->stream>>>(d_class_tot, n, K, fs.L, fs.L_len,
                                                            ctx->parent.as<double>());
    PD_CUDA(cudaGetLastError());
    ctx->launches++;
    fs.parent = ctx->parent.as<double>();
    fs.tiles = tiles;
    fs.out = static_cast<SplitOut *>(ctx->res_out);
    fs.out_cl = ctx->res_cl;
    fs.rechecked = ctx->res_recheck;
    fs.ord = d_ord;
  }
  HistGrid g;
  memset(&g, 0, sizeof(g));
  g.ds = devset(ctx);
  g.rec = d_rec;
  g.items = ctx->items.as<WorkItem>();
  g.n_items = n_big;
  g.tiles = tiles;
  for (int b = 0; b < 4; b++) {
    g.small[b].nc = kSmallRows[b];
    g.small[b].may = n_small[b] || (rank && split_slots && ctx->fuse_max && (b == 1 || (b == 3 && K > 8)) &&
                                    rank_smem(kSmallRows[b], T, span, small_threads(kSmallRows[b])) <= kRankSmemMax);
    g.small[b].n_items = n_small[b];
    g.small[b].smem = n_small[b] ? rank_smem(kSmallRows[b], T, span, small_threads(kSmallRows[b])) : 0;
  }
  g.cand_feat = ctx->cand_feat.ptr;
  g.cand_thr = ctx->cand_thr.ptr;
  g.hist = ctx->hist.as<uint32_t>();
  g.F = F;
  g.T = T;
  g.K = K;
  g.TP = rank ? 0 : padded_rows(T);
  g.thr_lo = p->thr_low;
  g.thr_span = span;
  g.smem = rank ? rank_smem(K, T, span, kRankThreads) : hist_smem(ctx, T, any_fused);
  g.fs = fs;
  g.ev_before = ev_before;
  g.queue = nullptr;
  if (persist && n_big * tiles < 0x7fffffffull) {
    PD_TRY(ctx->hist_queue.ensure(16));
    g.queue = ctx->hist_queue.as<unsigned>();
  }
  if constexpr (P::kRtcOnly) {
    PD_TRY(launch_hist_grid_rtc(ctx, g));
  } else {
    PD_TRY(launch_hist_grid<P>(ctx, g));
  }
  if (ev_after) PD_CUDA(cudaEventRecord(ev_after, ctx->stream));
  return PD_OK;
}

// Algorithmic HBM bytes of one histogram launch: the training-set images read
// once, 16 bytes per active sample (its SampleRec), the
// candidate table of every slot read once, and the K*T*F uint32 histogram
// written once for each slot whose split is not fused into the kernel.
static uint64_t hist_algorithmic_bytes(const pd_ctx *ctx, const pd_train_params *p, uint64_t n_samples,
                                       uint32_t n_slots, uint32_t n_written, uint64_t image_bytes) {
  const uint64_t F = p->n_features, T = p->n_thresholds, K = ctx->cfg.n_classes;
  const uint64_t fs = feat_size(ctx->cfg.feat_type);
  return image_bytes + (uint64_t)sizeof(SampleRec) * n_samples + (uint64_t)n_slots * (T * F * fs + ctx->cfg.feat_dim * F * fs) +
         (uint64_t)n_written * K * T * F * 4;
}

// Split kernels over n slots: slots[0..n) of the slice, or 0..n-1 when
// d_slot_list is null.
template <bool CUM>
static int launch_split(pd_ctx *ctx, const pd_train_params *p, uint32_t n, const uint32_t *d_hist,
                        const uint8_t *d_perm, const uint32_t *d_class_tot,
                        const uint32_t *d_slot_list = nullptr, uint32_t slice_slots = 0,
                        const uint32_t *d_ord = nullptr) {
  if (!n) return PD_OK;
  const uint32_t all = d_slot_list ? slice_slots : n;
  const uint32_t F = p->n_features;
  // Parts per node: enough CTAs to fill the GPU when the frontier is small.
  const uint32_t max_parts = (F + kSplitCols - 1) / kSplitCols;
  uint32_t parts = std::min<uint32_t>(max_parts, std::max<uint32_t>(1, (4 * 152 + n - 1) / n));
  uint32_t cols = (F + parts - 1) / parts;
  cols = (cols + 31) / 32 * 32;
  parts = (F + cols - 1) / cols;
  PD_TRY(ctx->split_scratch.ensure((size_t)all * 8 + (size_t)all * parts * sizeof(SplitPart) + 16));
  unsigned *node_max = ctx->split_scratch.as<unsigned>();
  PD_CUDA(cudaMemsetAsync(node_max, 0, (size_t)all * 8, ctx->stream));
  SplitArgs a;
  a.hist = d_hist;
  a.perm = d_perm;
  a.class_tot = d_class_tot;
  a.g32 = ctx->g32.as<float>();
  a.L = ctx->log2_tab.as<double>();
  a.L_len = ctx->log2_len;
  a.F = F;
  a.T = p->n_thresholds;
  a.K = ctx->cfg.n_classes;
  a.delta = recheck_delta(ctx->cfg.n_classes);
  a.cols = cols;
  a.parts = parts;
  a.node_max = node_max;
  a.done = node_max + all;
  a.part_best = reinterpret_cast<SplitPart *>(ctx->split_scratch.as<uint8_t>() + (size_t)all * 8);
  a.slot_list = d_slot_list;
  a.ord = d_ord;
  a.out = static_cast<SplitOut *>(ctx->res_out);
  a.out_cl = ctx->res_cl;
  a.rechecked = ctx->res_recheck;
  const dim3 grid(parts, n);
  auto run = [&]<int KM>() -> int {
    k_split_g32<KM, CUM><<<grid, kSplitCols, 0, ctx->stream>>>(a);
    k_split_pick<KM, CUM><<<grid, kSplitCols, 0, ctx->stream>>>(a);
    PD_CUDA(cudaGetLastError());
    ctx->launches += 2;
    return PD_OK;
  };
  // class loops are unrolled to KM >= K; the common class counts get exact KM
  const int K = ctx->cfg.n_classes;
  if (K <= 3) return run.template operator()<3>();
  if (K <= 4) return run.template operator()<4>();
  if (K <= 8) return run.template operator()<8>();
  if (K <= 9) return run.template operator()<9>();
  if (K <= 16) return run.template operator()<16>();
  if (K <= 21) return run.template operator()<21>();
  if (K <= 32) return run.template operator()<32>();
  return run.template operator()<64>();
}

static float elapsed(cudaEvent_t a, cudaEvent_t b) {
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  return ms;
}

// ------------------------------------------------------------- one tree ----
// A rank of candidate-sharded training: it evaluates candidates
// [f_base, f_base + params->n_features) of F_total, and `exchange` turns the
// ranks' best splits of a slice into the global ones.
struct Shard {
  uint32_t f_base, F_total;
  pd_exchange_fn exchange;
  void *user;
};

// Order key of a double (the device's gain_order_key).
static int64_t gain_key_host(double g) {
  int64_t b;
  memcpy(&b, &g, 8);
  return b < 0 ? (INT64_MIN - b - 1) : b;
}

// With `prop`, candidates f < n_prop of every node come from the proposal
// network (learned proposals); with ctx->collect_records, one pd_record per
// split node is kept; with `shard`, this rank's candidates are a range of the
// node's and each slice's winners are exchanged with the other ranks.
// One level of the training images' node map (k_node_map_step over every
// pixel, labelled pixels advancing) with the device tree being trained.
static int launch_node_map_step(pd_ctx *ctx, const int32_t *in, int32_t *out) {
  const RtcKernels *rk = nullptr;
  PD_TRY(rtc_kernels(ctx, &rk));
  NodeMapStep a;
  a.pixels = ctx->pixels.as<uint8_t>();
  a.img_off = ctx->img_off.as<uint64_t>();
  a.img_wh = ctx->img_wh.as<uint32_t>();
  a.map_off = ctx->nm_off.as<uint64_t>();
  a.n_images = ctx->n_images;
  a.n_pix = ctx->nm_pixels;
  a.mask = ctx->nm_label.as<uint8_t>();
  a.map_in = in;
  a.map_out = out;
  a.lc = ctx->t_lc.as<int32_t>();
  a.feat = ctx->t_feat.ptr;
  a.thr = ctx->t_thr.ptr;
  a.post = ctx->t_post.as<float>();
  a.n_classes = (uint32_t)ctx->cfg.n_classes;
  a.level = ctx->nm_level;
  a.n_nodes = ctx->nm_nodes;
  a.magic = ctx->magic_tab.as<uint32_t>();
  void *args[] = {&a};
  return rtc_launch(ctx, rk->node_map_step, dim3((unsigned)((a.n_pix + 255) / 256)), dim3(256), 0, args);
}

template <class P>
static int train_tree_impl(pd_ctx *ctx, const pd_train_params *p, uint32_t tree_id, uint32_t end_depth,
                           const float *root_prior, int32_t *lc, typename P::feat_t *feats,
                           typename P::feat_t *thrs, float *posts, pd_proposer *prop = nullptr,
                           uint32_t n_prop = 0, const Shard *shard = nullptr) {
  using FeatT = typename P::feat_t;
  constexpr int D = P::kFeatDim;
  const auto t_start = std::chrono::steady_clock::now();
  const uint32_t F = p->n_features, K = ctx->cfg.n_classes;
  const uint64_t n_nodes = (1ull << end_depth) - 1ull;
  const uint64_t S = ctx->n_samples;
  cudaStream_t st = ctx->stream;
  pd_train_stats stats;
  memset(&stats, 0, sizeof(stats));
  const uint64_t h2d0 = ctx->bytes_h2d, d2h0 = ctx->bytes_d2h, launches0 = ctx->launches;
  const uint64_t image_bytes = ctx->pixels_bytes;
  ctx->records.clear();

  PD_TRY(ensure_log2_table(ctx, S + 2));
  memcpy(posts, root_prior, sizeof(float) * K);
  if (ctx->tree_feature) {
    // A feature that reads the tree needs it on the device, as the caller holds it
    // (init:33-50); the trainer itself reads splits by frontier slot.
    PD_TRY(ctx->t_lc.ensure(n_nodes * 4));
    PD_TRY(ctx->t_feat.ensure(n_nodes * D * sizeof(FeatT)));
    PD_TRY(ctx->t_thr.ensure(n_nodes * sizeof(FeatT)));
    PD_TRY(ctx->t_post.ensure(n_nodes * K * 4));
    PD_CUDA(h2d(ctx, ctx->t_lc.ptr, lc, n_nodes * 4));
    PD_CUDA(h2d(ctx, ctx->t_feat.ptr, feats, n_nodes * D * sizeof(FeatT)));
    PD_CUDA(h2d(ctx, ctx->t_thr.ptr, thrs, n_nodes * sizeof(FeatT)));
    PD_CUDA(h2d(ctx, ctx->t_post.ptr, posts, n_nodes * K * 4));
  }

  PD_TRY(ctx->snode.ensure(S * 4 + 4));
  for (int b = 0; b < 2; b++) {
    PD_TRY(ctx->act[b].ensure(S * 4 + 4));
    PD_TRY(ctx->act_slot[b].ensure(S * 4 + 4));
    PD_TRY(ctx->act_rec[b].ensure(S * sizeof(SampleRec) + sizeof(SampleRec)));
  }
  PD_TRY(ctx->flags.ensure(S + 16));
  PD_TRY(ctx->scan_blocks.ensure((S / kScanItems + 4) * 8));
  PD_TRY(ctx->h_chk.ensure(16));
  PD_CUDA(cudaMemsetAsync(ctx->snode.ptr, 0, S * 4, st));
  // The regrouping of a level is checked at the next level's synchronisation.  Until
  // then a position it missed (a feature that is no function of its inputs) holds a
  // sample all the same: the first of the set, or one of an earlier level.  The
  // kernels before the check take any samples (samples_disagree).
  PD_CUDA(cudaMemsetAsync(ctx->act[1].ptr, 0, S * 4, st));
  PD_CUDA(cudaMemsetAsync(ctx->act_slot[1].ptr, 0, S * 4, st));
  PD_CUDA(cudaMemsetAsync(ctx->act_rec[1].ptr, 0, S * sizeof(SampleRec), st));
  if (ctx->tree_feature) {
    // every pixel starts at the root (traverse_ts.hpp:146-163 fills the node image with 0)
    PD_CHECK(ctx->nm_pixels, PD_ERR_STATE, "the training set was uploaded before the plugin was compiled");
    ctx->nm_cur = 0;
    ctx->nm_nodes = (int32_t)n_nodes;
    PD_CUDA(cudaMemsetAsync(ctx->nm_map[0].ptr, 0, ctx->nm_pixels * 4, st));
  }
  if (S) {
    k_iota<<<(unsigned)((S + 255) / 256), 256, 0, st>>>(ctx->act[0].as<uint32_t>(), ctx->act_slot[0].as<uint32_t>(), (uint32_t)S);
    k_gather_rec<<<(unsigned)((S + 255) / 256), 256, 0, st>>>(ctx->act[0].as<uint32_t>(), (uint32_t)S,
                                                               ctx->s_rec.as<SampleRec>(), ctx->act_rec[0].as<SampleRec>());
    ctx->launches += 2;
  }
  PD_CUDA(cudaGetLastError());

  // the frontier: nodes, class totals [slot][K], and their ranges of active samples
  std::vector<int32_t> frontier{0}, next;
  std::vector<uint32_t> tot(ctx->root_class_tot), next_tot;
  std::vector<uint64_t> cur_off{0, S}, next_off;
  int cur = 0;
  uint64_t n_act = S, pending = ~0ull;  // pending: samples the last regrouping must have placed (~0: none to check)
  uint32_t pending_depth = 0;
  // slices are sized for all F_total candidates when sharded, so every rank cuts the same slices
  pd_train_params p_all = *p;
  if (shard) p_all.n_features = shard->F_total;
  const uint64_t per_slot = slot_bytes(ctx, &p_all);
  const uint32_t max_slots = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(ctx->hist_budget / per_slot, 1u << 30));
  std::vector<SplitOut> h_out;
  std::vector<uint32_t> cr(K);
  std::vector<uint8_t> split_now;
  std::vector<uint32_t> left_cnt;  // left class counts of every slot of the level
  std::vector<FeatT> level_par;    // feature values and threshold of every slot of the level
  cudaEvent_t *ev = ctx->ev;
  // after a synchronisation: the last regrouping's counts, and its time
  auto check_regroup = [&]() -> int {
    if (pending == ~0ull) return PD_OK;
    const unsigned long long *chk = ctx->h_chk.as<unsigned long long>();
    const uint64_t want = pending, got = (chk[0] & 0xffffffffull) + (chk[0] >> 32);
    pending = ~0ull;
    PD_CHECK(chk[1] == 0 && got == want, PD_ERR_STATE,
             "reassignment disagrees with the split counts at depth %u (%llu vs %llu samples, %u misplaced)",
             pending_depth, (unsigned long long)got, (unsigned long long)want, (uint32_t)chk[1]);
    return PD_OK;
  };
  bool timed_reassign = false;
  auto after_sync = [&]() -> int {
    if (timed_reassign) stats.ms_reassign += elapsed(ev[4], ev[5]);
    timed_reassign = false;
    return check_regroup();
  };

  for (uint32_t depth = 1; depth < end_depth; depth++) {
    ctx->nm_level = (int32_t)depth - 1;  // the node map's level: the frontier's
    const uint32_t nf = (uint32_t)frontier.size();
    if (nf == 0) break;
    stats.evals += cur_off.back() * F;
    stats.nodes_trained += nf;
    const uint32_t cap = std::min(nf, max_slots);
    PD_TRY(ensure_slice(ctx, p, cap));
    split_now.assign(nf, 0);
    left_cnt.assign((size_t)nf * K, 0u);
    level_par.assign((size_t)nf * (D + 1), (FeatT)0);

    for (uint32_t s0 = 0; s0 < nf; s0 += cap) {
      const uint32_t ns = std::min(cap, nf - s0);
      // nodes and class totals of the slice, in one copy
      const size_t node_bytes = ((size_t)ns * 4 + 15) / 16 * 16;
      PD_TRY(ctx->h_pre.ensure(node_bytes + (size_t)ns * K * 4));
      PD_TRY(ctx->d_pre.ensure(node_bytes + (size_t)ns * K * 4));
      const uint32_t *ctot = &tot[(size_t)s0 * K];
      memcpy(ctx->h_pre.ptr, &frontier[s0], (size_t)ns * 4);
      memcpy(ctx->h_pre.as<uint8_t>() + node_bytes, ctot, (size_t)ns * K * 4);
      PD_CUDA(h2d(ctx, ctx->d_pre.ptr, ctx->h_pre.ptr, node_bytes + (size_t)ns * K * 4));
      const int32_t *d_nodes = ctx->d_pre.as<int32_t>();
      const uint32_t *d_ctot = reinterpret_cast<const uint32_t *>(ctx->d_pre.as<uint8_t>() + node_bytes);
      PD_TRY(set_results(ctx, ns));
      PD_CUDA(cudaMemsetAsync(ctx->res_recheck, 0, 16, st));
      std::vector<uint64_t> off(cur_off.begin() + s0, cur_off.begin() + s0 + ns + 1);
      PD_CUDA(cudaEventRecord(ev[0], st));
      const uint32_t *d_ord = nullptr;
      PropSrc src;
      if (prop) {
        // the network's mixture for every node of the slice, then the table drawn from it
        PD_TRY(proposer_infer(prop, d_ctot, ns, depth, n_prop, &src));
        PD_TRY(launch_candidates<P>(ctx, p, tree_id, d_nodes, ns, ctx->cand_order, &d_ord, &src));
      } else {
        PD_TRY(launch_candidates<P>(ctx, p, tree_id, d_nodes, ns, ctx->cand_order, &d_ord, nullptr,
                                    shard ? shard->f_base : 0u));
      }
      PD_CUDA(cudaEventRecord(ev[1], st));
      uint64_t n_items = 0;
      std::vector<uint32_t> split_slots;
      const uint32_t *d_split_list = nullptr;
      PD_TRY(launch_hist<P>(ctx, p, off.data(), ns, ctx->act_rec[cur].as<SampleRec>(), &n_items, ev[6], ev[2],
                            &split_slots, d_ctot, ctot, d_ord, prop ? &src : nullptr, &d_split_list));
      stats.hist_launches++;
      stats.hist_bytes += hist_algorithmic_bytes(ctx, p, off.back() - off.front(), ns, (uint32_t)split_slots.size(),
                                                 image_bytes);
      PD_TRY(launch_split<false>(ctx, p, (uint32_t)split_slots.size(), ctx->hist.as<uint32_t>(),
                                 ctx->cand_perm.as<uint8_t>(), d_ctot, d_split_list, ns, d_ord));
      // the winners' feature values and thresholds, from the candidate tables
      k_split_params<FeatT><<<(ns + 127) / 128, 128, 0, st>>>(
          static_cast<SplitOut *>(ctx->res_out), ns, ctx->cand_feat.as<FeatT>(), ctx->cand_thr.as<FeatT>(),
          ctx->cand_perm.as<uint8_t>(), p->n_features, p->n_thresholds, D, static_cast<FeatT *>(ctx->res_par));
      PD_CUDA(cudaGetLastError());
      ctx->launches++;
      PD_CUDA(cudaEventRecord(ev[3], st));
      PD_TRY(ctx->h_res.ensure(ctx->res_bytes));
      PD_CUDA(d2h(ctx, ctx->h_res.ptr, ctx->res_out, ctx->res_bytes));
      PD_CUDA(cudaStreamSynchronize(st));
      PD_TRY(after_sync());
      auto host = [&](const void *d) {  // where a result lies in the copy
        return ctx->h_res.as<uint8_t>() + (static_cast<const uint8_t *>(d) - static_cast<const uint8_t *>(ctx->res_out));
      };
      h_out.assign(reinterpret_cast<const SplitOut *>(host(ctx->res_out)),
                   reinterpret_cast<const SplitOut *>(host(ctx->res_out)) + ns);
      uint32_t *h_cl = &left_cnt[(size_t)s0 * K];
      FeatT *h_par = &level_par[(size_t)s0 * (D + 1)];
      memcpy(h_cl, host(ctx->res_cl), (size_t)ns * K * 4);
      memcpy(h_par, host(ctx->res_par), (size_t)ns * (D + 1) * sizeof(FeatT));
      unsigned long long rechecked[2];
      memcpy(rechecked, host(ctx->res_recheck), 16);
      PD_CHECK(rechecked[1] == 0, PD_ERR_STATE,
               "reassignment disagrees with the split counts: a node of depth %u has other samples than its class totals",
               depth);
      stats.ms_candidates += elapsed(ev[0], ev[1]);
      stats.ms_hist += elapsed(ev[6], ev[2]);
      stats.ms_split += elapsed(ev[2], ev[3]);
      stats.split_rechecked += rechecked[0];

      if (shard) {
        // the ranks' best splits -> the global ones: largest exact gain, ties to the lowest t * F + f
        std::vector<int64_t> key(ns), idx(ns);
        for (uint32_t i = 0; i < ns; i++) {
          const SplitOut &o = h_out[i];
          key[i] = o.t < 0 ? INT64_MIN : gain_key_host(o.gain);
          idx[i] = o.t < 0 ? -1 : (int64_t)o.t * shard->F_total + (int64_t)(shard->f_base + (uint32_t)o.f);
          if (o.t < 0) memset(&h_cl[(size_t)i * K], 0, K * 4);
        }
        PD_CHECK(shard->exchange(shard->user, ns, K, key.data(), idx.data(), h_cl) == 0, PD_ERR_STATE,
                 "the exchange of the ranks' best splits failed at depth %u", depth);
        for (uint32_t i = 0; i < ns; i++) {
          SplitOut &o = h_out[i];
          if (idx[i] < 0) {
            o.t = -1;
            continue;
          }
          const uint32_t t_g = (uint32_t)(idx[i] / shard->F_total), f_g = (uint32_t)(idx[i] % shard->F_total);
          const bool mine = o.t >= 0 && (uint32_t)o.t == t_g && shard->f_base + (uint32_t)o.f == f_g;
          o.t = (int32_t)t_g;
          o.gain = 0.0;
          if (!mine) {
            // the winner lives on another rank: its values from its seeds (hist_update.cl:62-184)
            const uint32_t node = (uint32_t)frontier[s0 + i];
            FeatT fv[PD_MAX_FEAT_DIM];
            candidate_feature<FeatT>(tree_id, node, f_g, D, p->feat_low, p->feat_up, fv);
            for (int d = 0; d < D; d++) h_par[(size_t)i * (D + 1) + d] = fv[d];
            h_par[(size_t)i * (D + 1) + D] = candidate_threshold<FeatT>(tree_id, node, f_g, t_g, p->thr_low, p->thr_up);
          }
        }
      }

      // finalize (learn_best_featthr.hpp:117-243)
      for (uint32_t i = 0; i < ns; i++) {
        const SplitOut &o = h_out[i];
        if (o.t < 0) continue;
        const uint32_t n = (uint32_t)frontier[s0 + i];
        const uint32_t *cl = h_cl + (size_t)i * K, *nt = ctot + (size_t)i * K;
        uint32_t lsum = 0, rsum = 0;
        for (uint32_t l = 0; l < K; l++) {
          cr[l] = nt[l] - cl[l];
          lsum += cl[l];
          rsum += cr[l];
        }
        if (!lsum || !rsum) continue;
        const uint64_t L = 2ull * n + 1, R = 2ull * n + 2;
        for (uint32_t l = 0; l < K; l++) {
          posts[L * K + l] = (float)cl[l] / (float)lsum;
          posts[R * K + l] = (float)cr[l] / (float)rsum;
        }
        lc[L] = -1;
        lc[R] = -1;
        // = candidate_feature / candidate_threshold of (o.f, o.t), read from the tables
        for (int d = 0; d < D; d++) feats[(size_t)n * D + d] = h_par[(size_t)i * (D + 1) + d];
        thrs[n] = h_par[(size_t)i * (D + 1) + D];
        lc[n] = (int32_t)L;
        split_now[s0 + i] = 1;
        stats.nodes_split++;
        if (ctx->collect_records) {
          pd_record r;
          memset(&r, 0, sizeof(r));
          r.depth = depth;
          r.count = lsum + rsum;
          r.node = n;
          r.tree = tree_id;
          r.gain = o.gain;
          for (int d = 0; d < D; d++) r.feat[d] = (int32_t)feats[(size_t)n * D + d];
          r.thr = (int32_t)thrs[n];
          for (uint32_t l = 0; l < K; l++) r.class_count[l] = nt[l];
          ctx->records.push_back(r);
        }
      }
    }

    if (ctx->tree_feature) {
      // device tree update for the frontier nodes and their children
      const uint64_t nmin = (uint64_t)frontier.front(), nmax = (uint64_t)frontier.back();
      const uint64_t cmax = std::min<uint64_t>(n_nodes - 1, 2 * nmax + 2);
      PD_CUDA(h2d(ctx, ctx->t_lc.as<int32_t>() + nmin, lc + nmin, (cmax - nmin + 1) * 4));
      PD_CUDA(h2d(ctx, ctx->t_feat.as<FeatT>() + nmin * D, feats + nmin * D, (nmax - nmin + 1) * D * sizeof(FeatT)));
      PD_CUDA(h2d(ctx, ctx->t_thr.as<FeatT>() + nmin, thrs + nmin, (nmax - nmin + 1) * sizeof(FeatT)));
      if (2 * nmin + 1 < n_nodes)
        PD_CUDA(h2d(ctx, ctx->t_post.as<float>() + (2 * nmin + 1) * K, posts + (2 * nmin + 1) * K,
                    (cmax - (2 * nmin + 1) + 1) * K * 4));
    }

    // next frontier (init:333-365: leaf children with more than perLeafSamplesThr samples)
    next.clear();
    next_tot.clear();
    next_off.assign(1, 0);
    const size_t sn_bytes = (size_t)nf * sizeof(SlotNext), par_bytes = (size_t)nf * (D + 1) * sizeof(FeatT);
    PD_TRY(ctx->h_splits.ensure(sn_bytes + par_bytes));
    PD_TRY(ctx->d_splits.ensure(sn_bytes + par_bytes));
    SlotNext *sn = ctx->h_splits.as<SlotNext>();
    long long base_l = 0, base_r = 0;
    const bool more = depth + 1 < end_depth;
    for (uint32_t i = 0; i < nf; i++) {
      SlotNext x;
      x.k_l = x.k_r = x.child = -1;
      x.beg = (uint32_t)next_off.back();
      x.adj_l = x.adj_r = 0;
      if (split_now[i]) {
        const uint64_t n = (uint64_t)frontier[i], L = 2 * n + 1, R = 2 * n + 2;
        const uint32_t *cl = &left_cnt[(size_t)i * K], *nt = &tot[(size_t)i * K];
        uint64_t lsum = 0;
        for (uint32_t l = 0; l < K; l++) lsum += cl[l];
        const uint64_t rsum = cur_off[i + 1] - cur_off[i] - lsum;
        x.child = (int32_t)L;
        if (more && lsum > p->per_leaf_samples_thr) {
          x.k_l = (int32_t)next.size();
          x.adj_l = (long long)next_off.back() - base_l;
          base_l += (long long)lsum;
          next.push_back((int32_t)L);
          next_off.push_back(next_off.back() + lsum);
          next_tot.insert(next_tot.end(), cl, cl + K);
        }
        if (more && rsum > p->per_leaf_samples_thr) {
          x.k_r = (int32_t)next.size();
          x.adj_r = (long long)next_off.back() - base_r;
          base_r += (long long)rsum;
          next.push_back((int32_t)R);
          next_off.push_back(next_off.back() + rsum);
          for (uint32_t l = 0; l < K; l++) next_tot.push_back(nt[l] - cl[l]);
        }
      }
      x.end = (uint32_t)next_off.back();
      x.mid = x.k_r >= 0 ? (uint32_t)next_off[x.k_r] : x.end;
      sn[i] = x;
    }
    // the level's splits by slot, in one copy
    memcpy(ctx->h_splits.as<uint8_t>() + sn_bytes, level_par.data(), par_bytes);
    PD_CUDA(h2d(ctx, ctx->d_splits.ptr, ctx->h_splits.ptr, sn_bytes + par_bytes));
    const SlotNext *d_next = ctx->d_splits.as<SlotNext>();
    const FeatT *d_par = reinterpret_cast<const FeatT *>(ctx->d_splits.as<uint8_t>() + sn_bytes);
    PD_CUDA(cudaEventRecord(ev[4], st));
    if (n_act && is_user_plugin(ctx)) {
      const RtcKernels *rk = nullptr;
      PD_TRY(rtc_kernels(ctx, &rk));
      DevSet ds = devset(ctx);
      const uint32_t *a_ = ctx->act[cur].as<uint32_t>(), *as_ = ctx->act_slot[cur].as<uint32_t>();
      const SampleRec *r_ = ctx->act_rec[cur].as<SampleRec>();
      uint32_t na = (uint32_t)n_act;
      int32_t *sn_ = ctx->snode.as<int32_t>();
      uint8_t *fl = ctx->flags.as<uint8_t>();
      void *args[] = {&ds, &a_, &r_, &as_, &na, &sn_, &d_par, &d_next, &fl};
      PD_TRY(rtc_launch(ctx, rk->reassign, dim3((unsigned)((n_act + 255) / 256)), dim3(256), 0, args));
    } else if constexpr (!P::kRtcOnly) {
      if (n_act) {
        k_reassign<P><<<(unsigned)((n_act + 255) / 256), 256, 0, st>>>(
            devset(ctx), ctx->act[cur].as<uint32_t>(), ctx->act_rec[cur].as<SampleRec>(),
            ctx->act_slot[cur].as<uint32_t>(), (uint32_t)n_act, ctx->snode.as<int32_t>(), d_par, d_next,
            ctx->flags.as<uint8_t>());
        PD_CUDA(cudaGetLastError());
        ctx->launches++;
      }
    }
    if (ctx->tree_feature && !next.empty()) {
      // the node map of the next depth, from this depth's map and the tree as it now stands
      PD_TRY(launch_node_map_step(ctx, ctx->nm_map[ctx->nm_cur].as<int32_t>(),
                                  ctx->nm_map[1 - ctx->nm_cur].as<int32_t>()));
      ctx->nm_cur = 1 - ctx->nm_cur;
    }
    const uint64_t n_next = next_off.back();
    if (!next.empty() && n_act) {
      const uint32_t nb = (uint32_t)((n_act + kScanItems - 1) / kScanItems);
      unsigned long long *bs = ctx->scan_blocks.as<unsigned long long>();
      k_scan_reduce<<<nb, 256, 0, st>>>(ctx->flags.as<uint8_t>(), (uint32_t)n_act, bs);
      k_scan_blocks<<<1, 1024, 0, st>>>(bs, nb, bs + nb);
      k_scatter<<<nb, 256, 0, st>>>(ctx->flags.as<uint8_t>(), (uint32_t)n_act, bs, ctx->act[cur].as<uint32_t>(),
                                    ctx->act_slot[cur].as<uint32_t>(), d_next,
                                    ctx->act[1 - cur].as<uint32_t>(), ctx->act_slot[1 - cur].as<uint32_t>(),
                                    ctx->act_rec[cur].as<SampleRec>(), ctx->act_rec[1 - cur].as<SampleRec>(),
                                    bs + nb + 1);
      PD_CUDA(cudaGetLastError());
      ctx->launches += 3;
      PD_CUDA(d2h(ctx, ctx->h_chk.ptr, bs + nb, 16));  // checked after the next synchronisation
      pending = n_next;
      pending_depth = depth;
      cur = 1 - cur;
    }
    PD_CUDA(cudaEventRecord(ev[5], st));
    timed_reassign = true;
    n_act = n_next;
    frontier.swap(next);
    cur_off.swap(next_off);
    tot.swap(next_tot);
  }
  PD_CUDA(cudaStreamSynchronize(st));
  PD_TRY(after_sync());
  stats.ms_total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
  stats.h2d_bytes = ctx->bytes_h2d - h2d0;
  stats.d2h_bytes = ctx->bytes_d2h - d2h0;
  stats.kernel_launches = ctx->launches - launches0;
  ctx->stats = stats;
  return PD_OK;
}

}  // namespace pd

using namespace pd;

extern "C" int pd_train_tree(pd_ctx *ctx, const pd_train_params *params, uint32_t tree_id, uint32_t start_depth,
                             uint32_t end_depth, const float *root_prior, int32_t *left_child, void *features,
                             void *thresholds, float *posteriors) {
  PD_CHECK(ctx, PD_ERR_INVALID, "null context");
  PD_CHECK(ctx->have_dataset, PD_ERR_STATE, "no dataset uploaded");
  PD_CHECK(start_depth == 1, PD_ERR_INVALID, "Starting depth must be equal to 1");
  PD_CHECK(end_depth >= 1 && end_depth <= 24, PD_ERR_UNSUPPORTED, "end_depth %u outside [1,24]", end_depth);
  PD_CHECK(root_prior && left_child && features && thresholds && posteriors, PD_ERR_INVALID, "null tree array");
  PD_TRY(check_params(ctx, params));
  PD_CUDA(cudaSetDevice(ctx->device));
  return dispatch_config(ctx->cfg, [&]<class P>() {
    using FeatT = typename P::feat_t;
    return train_tree_impl<P>(ctx, params, tree_id, end_depth, root_prior, left_child,
                              static_cast<FeatT *>(features), static_cast<FeatT *>(thresholds), posteriors);
  });
}

extern "C" int pd_train_tree_proposed(pd_ctx *ctx, pd_proposer *prop, const pd_train_params *params,
                                      uint32_t n_proposed, uint32_t tree_id, uint32_t start_depth, uint32_t end_depth,
                                      const float *root_prior, int32_t *left_child, void *features, void *thresholds,
                                      float *posteriors) {
  PD_CHECK(ctx && prop, PD_ERR_INVALID, "null context or proposer");
  PD_CHECK(ctx->have_dataset, PD_ERR_STATE, "no dataset uploaded");
  PD_CHECK(start_depth == 1, PD_ERR_INVALID, "Starting depth must be equal to 1");
  PD_CHECK(end_depth >= 1 && end_depth <= 24, PD_ERR_UNSUPPORTED, "end_depth %u outside [1,24]", end_depth);
  PD_CHECK(root_prior && left_child && features && thresholds && posteriors, PD_ERR_INVALID, "null tree array");
  PD_TRY(check_params(ctx, params));
  PD_CHECK(n_proposed <= params->n_features, PD_ERR_INVALID, "n_proposed %u above n_features %u", n_proposed,
           params->n_features);
  PD_CUDA(cudaSetDevice(ctx->device));
  return dispatch_config(ctx->cfg, [&]<class P>() {
    using FeatT = typename P::feat_t;
    return train_tree_impl<P>(ctx, params, tree_id, end_depth, root_prior, left_child,
                              static_cast<FeatT *>(features), static_cast<FeatT *>(thresholds), posteriors, prop,
                              n_proposed);
  });
}

extern "C" int pd_train_tree_sharded(pd_ctx *ctx, const pd_train_params *params, uint32_t f_begin, uint32_t f_end,
                                     pd_exchange_fn exchange, void *user, uint32_t tree_id, uint32_t start_depth,
                                     uint32_t end_depth, const float *root_prior, int32_t *left_child, void *features,
                                     void *thresholds, float *posteriors) {
  PD_CHECK(ctx && exchange, PD_ERR_INVALID, "null context or exchange function");
  PD_CHECK(ctx->have_dataset, PD_ERR_STATE, "no dataset uploaded");
  PD_CHECK(start_depth == 1, PD_ERR_INVALID, "Starting depth must be equal to 1");
  PD_CHECK(end_depth >= 1 && end_depth <= 24, PD_ERR_UNSUPPORTED, "end_depth %u outside [1,24]", end_depth);
  PD_CHECK(root_prior && left_child && features && thresholds && posteriors, PD_ERR_INVALID, "null tree array");
  PD_TRY(check_params(ctx, params));
  PD_CHECK(f_begin < f_end && f_end <= params->n_features, PD_ERR_INVALID,
           "candidate range [%u, %u) outside [0, %u)", f_begin, f_end, params->n_features);
  PD_CUDA(cudaSetDevice(ctx->device));
  pd_train_params local = *params;
  local.n_features = f_end - f_begin;
  const Shard shard{f_begin, params->n_features, exchange, user};
  return dispatch_config(ctx->cfg, [&]<class P>() {
    using FeatT = typename P::feat_t;
    return train_tree_impl<P>(ctx, &local, tree_id, end_depth, root_prior, left_child, static_cast<FeatT *>(features),
                              static_cast<FeatT *>(thresholds), posteriors, nullptr, 0, &shard);
  });
}

extern "C" int pd_train_records(pd_ctx *ctx, pd_record *out, uint64_t cap, uint64_t *n) {
  PD_CHECK(ctx && n, PD_ERR_INVALID, "null argument");
  *n = ctx->records.size();
  if (out) memcpy(out, ctx->records.data(), std::min<uint64_t>(cap, ctx->records.size()) * sizeof(pd_record));
  return PD_OK;
}

extern "C" int pd_train_get_stats(pd_ctx *ctx, pd_train_stats *out) {
  PD_CHECK(ctx && out, PD_ERR_INVALID, "null argument");
  *out = ctx->stats;
  return PD_OK;
}

extern "C" int pd_train_sample_nodes(pd_ctx *ctx, int32_t *out) {
  PD_CHECK(ctx && out, PD_ERR_INVALID, "null argument");
  PD_CHECK(ctx->have_dataset && ctx->snode.cap >= ctx->n_samples * 4, PD_ERR_STATE, "no training run");
  PD_CUDA(cudaSetDevice(ctx->device));
  PD_CUDA(d2h(ctx, out, ctx->snode.ptr, ctx->n_samples * 4));
  PD_CUDA(cudaStreamSynchronize(ctx->stream));
  return PD_OK;
}

// ------------------------------------------------------ stage entry points ----
extern "C" int pd_candidates(pd_ctx *ctx, const pd_train_params *params, uint32_t tree_id, const int32_t *nodes,
                             uint32_t n_nodes, void *features_out, void *thresholds_out) {
  PD_CHECK(ctx && nodes && features_out && thresholds_out, PD_ERR_INVALID, "null argument");
  PD_TRY(check_params(ctx, params));
  PD_CUDA(cudaSetDevice(ctx->device));
  return dispatch_config(ctx->cfg, [&]<class P>() {
    using FeatT = typename P::feat_t;
    constexpr int D = P::kFeatDim;
    const uint32_t F = params->n_features, T = params->n_thresholds;
    PD_TRY(ensure_slice(ctx, params, n_nodes));
    DevBuf dn;
    PD_TRY(dn.ensure((size_t)n_nodes * 4));
    PD_CUDA(h2d(ctx, dn.ptr, nodes, (size_t)n_nodes * 4));
    PD_TRY(launch_candidates<P>(ctx, params, tree_id, dn.as<int32_t>(), n_nodes));
    std::vector<FeatT> f((size_t)n_nodes * D * F), t((size_t)n_nodes * T * F);
    std::vector<uint8_t> perm((size_t)n_nodes * T * F);
    PD_CUDA(d2h(ctx, f.data(), ctx->cand_feat.ptr, f.size() * sizeof(FeatT)));
    PD_CUDA(d2h(ctx, t.data(), ctx->cand_thr.ptr, t.size() * sizeof(FeatT)));
    PD_CUDA(d2h(ctx, perm.data(), ctx->cand_perm.ptr, perm.size()));
    PD_CUDA(cudaStreamSynchronize(ctx->stream));
    dn.release();
    FeatT *fo = static_cast<FeatT *>(features_out), *to = static_cast<FeatT *>(thresholds_out);
    for (uint32_t n = 0; n < n_nodes; n++)
      for (uint32_t ff = 0; ff < F; ff++) {
        for (int d = 0; d < D; d++) fo[((size_t)n * F + ff) * D + d] = f[((size_t)n * D + d) * F + ff];
        for (uint32_t j = 0; j < T; j++) {
          const size_t src = ((size_t)n * T + j) * F + ff;
          to[((size_t)n * F + ff) * T + perm[src]] = t[src];
        }
      }
    return PD_OK;
  });
}

extern "C" int pd_hist(pd_ctx *ctx, const pd_train_params *params, uint32_t tree_id, const int32_t *sample_node,
                       const int32_t *nodes, uint32_t n_nodes, uint32_t *hist_out) {
  PD_CHECK(ctx && sample_node && nodes && hist_out, PD_ERR_INVALID, "null argument");
  PD_CHECK(ctx->have_dataset, PD_ERR_STATE, "no dataset uploaded");
  PD_CHECK(!ctx->tree_feature, PD_ERR_UNSUPPORTED,
           "the feature reads the tree and the node map, which only pd_train_tree keeps: no stage call");
  PD_TRY(check_params(ctx, params));
  PD_CUDA(cudaSetDevice(ctx->device));
  const uint64_t S = ctx->n_samples;
  const uint32_t F = params->n_features, T = params->n_thresholds, K = ctx->cfg.n_classes;
  // group samples by slot (stable)
  std::vector<std::pair<int32_t, uint32_t>> map(n_nodes);
  for (uint32_t i = 0; i < n_nodes; i++) map[i] = {nodes[i], i};
  std::sort(map.begin(), map.end());
  std::vector<uint64_t> cnt(n_nodes + 1, 0);
  std::vector<int64_t> slot_of(S, -1);
  for (uint64_t s = 0; s < S; s++) {
    auto it = std::lower_bound(map.begin(), map.end(), std::make_pair(sample_node[s], 0u));
    if (it != map.end() && it->first == sample_node[s]) {
      slot_of[s] = it->second;
      cnt[it->second + 1]++;
    }
  }
  for (uint32_t i = 0; i < n_nodes; i++) cnt[i + 1] += cnt[i];
  std::vector<uint32_t> act(cnt[n_nodes]);
  std::vector<uint64_t> pos(cnt.begin(), cnt.end() - 1);
  for (uint64_t s = 0; s < S; s++)
    if (slot_of[s] >= 0) act[pos[slot_of[s]]++] = (uint32_t)s;
  return dispatch_config(ctx->cfg, [&]<class P>() {
    PD_TRY(ensure_slice(ctx, params, n_nodes));
    DevBuf dn, da, drec, dref;
    PD_TRY(dn.ensure((size_t)n_nodes * 4));
    PD_TRY(da.ensure(act.size() * 4 + 4));
    PD_TRY(drec.ensure(act.size() * sizeof(SampleRec) + sizeof(SampleRec)));
    PD_TRY(dref.ensure((size_t)n_nodes * K * T * F * 4 + 4));
    PD_CUDA(h2d(ctx, dn.ptr, nodes, (size_t)n_nodes * 4));
    if (!act.empty()) {
      PD_CUDA(h2d(ctx, da.ptr, act.data(), act.size() * 4));
      k_gather_rec<<<(unsigned)((act.size() + 255) / 256), 256, 0, ctx->stream>>>(
          da.as<uint32_t>(), (uint32_t)act.size(), ctx->s_rec.as<SampleRec>(), drec.as<SampleRec>());
      PD_CUDA(cudaGetLastError());
      ctx->launches++;
    }
    PD_TRY(launch_candidates<P>(ctx, params, tree_id, dn.as<int32_t>(), n_nodes));
    uint64_t n_items = 0;
    PD_TRY(launch_hist<P>(ctx, params, cnt.data(), n_nodes, drec.as<SampleRec>(), &n_items));
    const uint64_t total = (uint64_t)n_nodes * K * F;
    if (total) {
      k_hist_to_ref<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>(
          ctx->hist.as<uint32_t>(), ctx->cand_perm.as<uint8_t>(), dref.as<uint32_t>(), n_nodes, K, T, F);
      PD_CUDA(cudaGetLastError());
    }
    PD_CUDA(d2h(ctx, hist_out, dref.ptr, (size_t)n_nodes * K * T * F * 4));
    PD_CUDA(cudaStreamSynchronize(ctx->stream));
    return PD_OK;
  });
}

extern "C" int pd_split(pd_ctx *ctx, const pd_train_params *params, const uint32_t *hist, const uint32_t *class_tot,
                        uint32_t n_nodes, int32_t *out_t, int32_t *out_f, double *out_gain) {
  PD_CHECK(ctx && hist && class_tot && out_t && out_f && out_gain, PD_ERR_INVALID, "null argument");
  PD_TRY(check_params(ctx, params));
  PD_CUDA(cudaSetDevice(ctx->device));
  const uint32_t F = params->n_features, T = params->n_thresholds, K = ctx->cfg.n_classes;
  uint64_t maxn = 2;
  for (uint32_t i = 0; i < n_nodes; i++) {
    uint64_t N = 0;
    for (uint32_t l = 0; l < K; l++) N += class_tot[(size_t)i * K + l];
    maxn = std::max(maxn, N + 2);
  }
  PD_TRY(ensure_log2_table(ctx, maxn));
  PD_TRY(ensure_slice(ctx, params, n_nodes));
  DevBuf dh, dc;
  PD_TRY(dh.ensure((size_t)n_nodes * K * T * F * 4 + 4));
  PD_TRY(dc.ensure((size_t)n_nodes * K * 4 + 4));
  PD_CUDA(h2d(ctx, dh.ptr, hist, (size_t)n_nodes * K * T * F * 4));
  PD_CUDA(h2d(ctx, dc.ptr, class_tot, (size_t)n_nodes * K * 4));
  PD_CUDA(cudaMemsetAsync(ctx->res_recheck, 0, 16, ctx->stream));
  PD_TRY(launch_split<true>(ctx, params, n_nodes, dh.as<uint32_t>(), nullptr, dc.as<uint32_t>()));
  std::vector<SplitOut> o(n_nodes);
  PD_CUDA(d2h(ctx, o.data(), ctx->res_out, n_nodes * sizeof(SplitOut)));
  PD_CUDA(cudaStreamSynchronize(ctx->stream));
  for (uint32_t i = 0; i < n_nodes; i++) {
    out_t[i] = o[i].t;
    out_f[i] = o[i].f;
    out_gain[i] = o[i].gain;
  }
  return PD_OK;
}

extern "C" int pd_log2_table(pd_ctx *ctx, uint32_t n, double *out) {
  PD_CHECK(ctx && out, PD_ERR_INVALID, "null argument");
  PD_CUDA(cudaSetDevice(ctx->device));
  PD_TRY(ensure_log2_table(ctx, n));
  PD_CUDA(d2h(ctx, out, ctx->log2_tab.ptr, (size_t)n * 8));
  PD_CUDA(cudaStreamSynchronize(ctx->stream));
  return PD_OK;
}
