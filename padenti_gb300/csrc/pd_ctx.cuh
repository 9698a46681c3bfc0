// Internal state of a pd_ctx: the device-resident training set, the training
// scratch buffers and the forest.
#pragma once

#include <vector>

#include "pd_common.cuh"

// Samples per iteration of the histogram kernel the tuning accepts (2, 4 or 8).
inline bool valid_hist_spi(uint32_t spi) { return spi == 2 || spi == 4 || spi == 8; }

namespace pd {
struct RtcPlugin;  // pd_rtc.cu
}

struct pd_ctx {
  pd_config cfg{};
  int device = 0;
  pd::RtcPlugin *rtc = nullptr;  // the compiled user feature plugin (PD_PLUGIN_USER)
  bool tree_feature = false;     // its computeFeature reads the tree: the node map is kept
  cudaStream_t stream = nullptr;
  // the small-node histogram launches of a level run beside its k_hist: forked from
  // stream, joined to it before anything else is enqueued (pd_hist_grid.cuh)
  cudaStream_t hist_side[4] = {};
  cudaEvent_t hist_fork = nullptr, hist_join[4] = {};
  uint64_t hist_budget = 8ull << 30;
  uint32_t chunk = 16384;  // samples per histogram work item (at most 65535)
  uint32_t hist_spi = 8;  // samples per iteration of the histogram kernel (2, 4 or 8)
  uint32_t fuse_max = 4096;  // nodes with at most this many samples get the fused split
  bool cand_order = true;    // order each node's candidate columns by first-probe offset
  bool cand_regs = true;     // candidate keys sorted in registers (T <= 64), else in shared memory
  bool persist = false;      // one persistent histogram grid per launch, items pulled largest first
  int upload_copy = 1;       // bulk inputs from pinned host memory: 0 copy engine, 1 SM copy kernel
  int n_sms = 0;             // multiprocessors of the context's GPU
  uint64_t sample_group = 512ull << 20;  // bytes of images + labels pd_sample stages per round trip
  bool collect_records = false;          // keep a pd_record per split node (learned proposals)
  std::vector<pd_record> records;        // of the last training call

  // ---- training set in HBM (cl_tree_trainer_impl_init.hpp:99-154 streams it
  // image by image; here it stays resident) ----
  bool have_dataset = false;
  uint32_t n_images = 0;
  uint64_t n_samples = 0;
  pd::DevBuf pixels;    // concatenated images
  uint64_t pixels_bytes = 0;
  pd::DevBuf img_off;   // uint64 byte offsets
  pd::DevBuf img_wh;    // uint32 w | h << 16
  pd::DevBuf s_xy;      // uint32 x | y << 16 per sample
  pd::DevBuf s_img;     // uint32 image per sample
  pd::DevBuf s_label;   // uint8 class (0..K-1) per sample
  std::vector<uint32_t> root_class_tot;  // samples per class (the root's class totals)
  pd_upload_stats upload_stats{};        // of the last pd_dataset_upload
  pd::HostBuf h_stage;           // pinned staging of the per-sample upload arrays
  pd::HostBuf h_items;           // pinned staging of a histogram launch's work list, zero and split slots
  // pinned staging of a frontier slice (nodes, class totals) and of a level's splits
  // (SlotNext, parameters), the results of a slice, the reassignment's check
  pd::HostBuf h_pre, h_splits, h_res, h_chk;
  pd::DevBuf d_pre, d_splits;
  pd::DevBuf log2_tab;  // double log2(n), n < log2_len
  pd::DevBuf xlog2_tab; // float c*log2(c), c < min(log2_len, 65536): the fused split's filter
  pd::DevBuf parent;    // [slots] parent term of the exact gain, for the fused split
  pd::DevBuf magic_tab; // uint32 RoundDiv multiplier by depth value (65536)
  uint64_t log2_len = 0;

  // ---- training scratch ----
  pd::DevBuf snode;                  // int32 node per sample
  pd::DevBuf act[2], act_slot[2];    // active samples sorted by frontier slot
  pd::DevBuf act_rec[2];             // their SampleRec, in the same order
  pd::DevBuf s_rec;                  // SampleRec of every uploaded sample
  pd::DevBuf flags;                  // uint8 per active sample
  pd::DevBuf scan_blocks;            // uint64 per scan block
  pd::DevBuf cand_feat, cand_thr, cand_perm;
  pd::DevBuf cand_ord;       // [slots][F] original candidate index of each column
  pd::DevBuf hist, g32;
  pd::DevBuf items, hist_queue;  // work list, slots to zero, slots to split
  // Results of a slice in one buffer, for one copy back: SplitOut [n], left class
  // counts [n][K], feature values and threshold [n][D + 1], rechecked candidates and
  // the report of samples_disagree (set_results).
  pd::DevBuf split_res;
  void *res_out = nullptr, *res_par = nullptr;
  uint32_t *res_cl = nullptr;
  unsigned long long *res_recheck = nullptr;
  size_t res_bytes = 0;
  pd::DevBuf split_scratch, fused_scratch;
  pd::DevBuf t_lc, t_feat, t_thr, t_post;  // device copy of the tree being trained
  // ---- node map of features that read the tree (tree_feature) ----
  pd::DevBuf nm_map[2];   // int32 node per pixel of every training image, this depth's and the next
  pd::DevBuf nm_off;      // uint64 [n_images + 1] first pixel of each image in the map
  pd::DevBuf nm_label;    // uint8 label of every pixel (nonzero: the map advances there)
  uint64_t nm_pixels = 0;
  int nm_cur = 0;
  int32_t nm_level = 0, nm_nodes = 0;  // the map's level (the depth being trained), the tree's node count
  pd::DevBuf np_map[2], np_desc;  // prediction: the map of the images predicted, their descriptors
  pd_train_stats stats{};

  // ---- forest (CLClassifier) ----
  std::vector<uint32_t> tree_depth;
  std::vector<uint64_t> tree_off;
  std::vector<int32_t> h_lc;
  std::vector<uint8_t> h_feat, h_thr;  // FeatType bytes
  std::vector<float> h_post;
  bool forest_dirty = true;
  pd::DevBuf f_lc, f_feat, f_thr, f_post, f_meta;
  pd::DevBuf f_cand;                   // FastNode or NodeRec of every forest node
  pd::DevBuf f_post4;                  // posterior rows padded to four classes a word, where K % 4 (k_pad_posteriors)
  pd::DevBuf f_gen;                    // NodeRec beside FastNode, for images past the fast form's sides
  uint64_t cand_version = ~0ull;       // forest_version f_cand was built for
  uint64_t gen_version = ~0ull;        // forest_version f_gen was built for
  bool forest_fast = false;            // every node takes the plugin's fast path (built-in plugins)
  pd::DevBuf p_img, p_mask, p_out;     // staging for host-buffer prediction
  uint64_t forest_version = 0;         // bumped when the forest arrays are uploaded again
  // mixed-size prediction batches: buffers, the layout they were built for and
  // the graph of the batch kernel (pd_predict_posterior_batch)
  pd::DevBuf b_img, b_mask, b_out, b_desc;
  std::vector<uint64_t> batch_key;
  cudaGraphExec_t batch_graph = nullptr;

  // ---- pixel samplers (pd_sample*) ----
  pd::DevBuf sm_desc;            // SampImage per image, item -> image map, checksums, counts, error
  pd::DevBuf sm_counts, sm_draws, sm_slots;  // class-weighted: segment counts, MT19937 outputs (reserve_draws), buckets
  pd::HostBuf h_sm_desc;         // pinned staging of the descriptors
  // pd_sample's two pipeline slots: a group is staged into one while the device
  // works on the other's (pinned data, descriptors, results; device copies; events
  // around the scan, the draws and the results)
  struct SampSlot {
    pd::HostBuf h_data, h_desc, h_out;
    pd::DevBuf d_data, d_desc, d_out;
    cudaEvent_t ev[4] = {};
  } samp[2];
  pd_sample_stats sample_stats{};
  // ---- label images (pd_rgb_to_labels*) ----
  pd::DevBuf lab_tab, lab_src, lab_dst;
  pd::HostBuf h_lab;

  cudaEvent_t ev[8] = {};
  uint64_t bytes_h2d = 0, bytes_d2h = 0, launches = 0;
};

namespace pd {
// Lets launches of a kernel take `smem` bytes of dynamic shared memory.  The limit is a
// property of the function, shared by every context of the process, and calls of
// several contexts may run at once: it is raised to the device's maximum and never to a
// launch's own size, which another thread's smaller launch would take away between the
// call and the launch.  It is a permission: occupancy follows from what a launch asks
// for.  Every kernel may take 32 KB (48 less its static arrays) without.
template <typename Kernel>
int allow_smem(const pd_ctx *c, Kernel *kernel, size_t smem) {
  if (smem <= 32768) return PD_OK;
  const void *fn = reinterpret_cast<const void *>(kernel);
  cudaFuncAttributes fa;
  PD_CUDA(cudaFuncGetAttributes(&fa, fn));
  int most = 0;
  PD_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  most -= (int)fa.sharedSizeBytes;
  PD_CHECK(smem <= (size_t)most, PD_ERR_CUDA, "a kernel needs %zu bytes of shared memory; the GPU offers %d", smem, most);
  if (fa.maxDynamicSharedSizeBytes < most)
    PD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  return PD_OK;
}
// Counted copies on the context stream.
inline cudaError_t h2d(pd_ctx *c, void *dst, const void *src, size_t n) {
  c->bytes_h2d += n;
  return cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, c->stream);
}
inline cudaError_t d2h(pd_ctx *c, void *dst, const void *src, size_t n) {
  c->bytes_d2h += n;
  return cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, c->stream);
}
}  // namespace pd

namespace pd {
struct PropSrc;
// The proposal network's mixture for n frontier nodes of depth `depth` (class
// totals d_ctot [n][K] on the device), on the context's stream (pd_propose.cu).
int proposer_infer(pd_proposer *p, const uint32_t *d_ctot, uint32_t n, uint32_t depth, uint32_t n_prop, PropSrc *src);
int ensure_log2_table(pd_ctx *ctx, uint64_t n);
// Whether the histogram kernels of a training call take the rank-table form (pd_train.cu).
bool rank_form(const pd_ctx *ctx, const pd_train_params *p, const PropSrc *prop = nullptr);
// Host -> device copy of bulk inputs on the context's stream (pd_api.cu).
int upload_bytes(pd_ctx *ctx, void *dst, const void *src, size_t n);
int init_tables(pd_ctx *ctx);
// Prepares the uploaded images for the plugin's eval_train (zero depths).
int map_training_pixels(pd_ctx *ctx, uint64_t bytes);
// The SampleRec of every uploaded sample (after map_training_pixels).
int build_sample_records(pd_ctx *ctx, uint64_t n_samples);
}
