// Forest prediction kernels: one thread per pixel walks every tree of the
// forest (cl_classifier_impl.hpp:478-552, predict.cl:36-117).  A header so that
// the kernels also compile, through NVRTC, for a user feature plugin.
#pragma once

#include "pd_plugins.cuh"

namespace pd {

struct TreeMeta {
  unsigned long long off;  // first node of the tree in the forest arrays
  uint32_t depth, pad;
};

// One forest node as the prediction kernels read it: the plugin's candidate
// record (P::candidate of its features, built once per forest upload), its
// threshold and its left child, together in one 16-byte-aligned record -- one
// visit fetches one or two 32-byte sectors instead of three arrays.
template <class P>
struct __align__(16) NodeRec {
  typename P::Cand c;
  typename P::feat_t thr;
  int32_t lc;
};

// The record of a forest all of whose nodes take the plugin's fast form: its
// constants there (one word per offset), threshold and left child, in one 16- or
// 32-byte record, so that a visit fetches one sector.
template <class P>
struct __align__(sizeof(typename P::FastCand) <= 8 ? 16 : 32) FastNode {
  typename P::FastCand c;
  int32_t thr, lc;
};
// What a kernel reads per node: a FastNode (AF) or a NodeRec.
template <class P, bool AF>
struct NodeOf {
  using type = NodeRec<P>;
};
template <class P>
struct NodeOf<P, true> {
  using type = FastNode<P>;
};
template <class P, bool AF>
using Node = typename NodeOf<P, AF>::type;

constexpr int kPredX = 32, kPredY = 8, kPredThreads = kPredX * kPredY;

// A record by 16-byte read-only loads (one 32-byte load was 6 % slower: L1 returns
// 128 bytes a cycle, and the last 8 of a FastNode are not wanted).
template <class N>
PD_D N load_node(const N *p) {
  static_assert(sizeof(N) % 16 == 0, "whole 16-byte words");
  N n;
  uint4 *d = reinterpret_cast<uint4 *>(&n);
#pragma unroll
  for (uint32_t i = 0; i < sizeof(N) / 16; i++) d[i] = ldg(reinterpret_cast<const uint4 *>(p) + i);
  return n;
}

// One pixel as the walks read it.
// AF: every node of the forest takes the plugin's fast form (P::fast, checked once
// per forest upload): the walk evaluates it from the pixel's words, with no
// per-visit test or slow path.
template <class P, bool AF>
struct Pixel {
  typename P::Prep prep;
  PD_D Pixel(const ImageRef<typename P::img_t> &im, int32_t x, int32_t y) : prep(P::prepare(im, x, y)) {}
  PD_D typename P::feat_t eval(const NodeRec<P> &n) const {
    return P::fast(n.c) ? P::template eval<true>(prep, n.c) : P::template eval<false>(prep, n.c);
  }
};
template <class P>
struct Pixel<P, true> {
  uint4 a, b;
  PD_D Pixel(const ImageRef<typename P::img_t> &im, int32_t x, int32_t y) {
    uint32_t pre[2] = {0u, 0u}, w[8];
    P::preload(im, x, y, pre);
    P::fast_words(im, x, y, pre, w);
    a = make_uint4(w[0], w[1], w[2], 0u);
    b = make_uint4(w[4], w[5], w[6], w[7]);
  }
  PD_D typename P::feat_t eval(const FastNode<P> &n) const { return P::template eval_fast<false>(a, b, n.c); }
};

// Leaf reached by one tree from the root (nodes: the tree's records).
template <class P, bool AF>
PD_D int32_t walk(const Pixel<P, AF> &px, const Node<P, AF> *__restrict__ nodes, uint32_t depth) {
  int32_t node = 0;
  for (uint32_t d = 1; d < depth; d++) {
    const Node<P, AF> n = load_node(nodes + node);
    if (n.lc < 0) break;  // leaf (-1); an untrained root (-2) also stops
    node = n.lc + (px.eval(n) <= n.thr ? 0 : 1);
  }
  return node;
}

// The record of every forest node, for the prediction kernels.
template <class P>
__global__ void k_forest_nodes(const typename P::feat_t *__restrict__ feat, const typename P::feat_t *__restrict__ thr,
                               const int32_t *__restrict__ lc, unsigned long long n_nodes,
                               NodeRec<P> *__restrict__ out) {
  const unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  if (i < n_nodes) {
    NodeRec<P> r;
    r.c = P::candidate(feat + i * P::kFeatDim);
    r.thr = thr[i];
    r.lc = lc[i];
    out[i] = r;
  }
}

// The FastNode of every forest node; sets *any_slow when a node needs the
// plugin's slow path (the NodeRec form is built then).
template <class P>
__global__ void k_forest_fast(const typename P::feat_t *__restrict__ feat, const typename P::feat_t *__restrict__ thr,
                              const int32_t *__restrict__ lc, unsigned long long n_nodes, FastNode<P> *__restrict__ out,
                              int *__restrict__ any_slow) {
  const unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  if (i >= n_nodes) return;
  const typename P::feat_t *f = feat + i * P::kFeatDim;
  FastNode<P> n;
  n.c = P::fast_candidate(f);
  n.thr = (int32_t)thr[i];
  n.lc = lc[i];
  out[i] = n;
  if (!P::fast(P::candidate(f))) *any_slow = 1;
}

// What bounds it (60 640x480 maps, 3 trees of depth 16, 9 classes): the L1 data pipe
// (90 %, 15 wavefronts per node visit: 24 bytes of record per lane, and probes that
// scatter once the lanes' nodes differ), then issue (81 %, 50 instructions per visit;
// 81 with the general records).  160 maps: 5.88 -> 3.97 ms.  CTA rows of 32 pixels:
// warps of 16x2 and 8x4 pixels were 9 and 28 % slower (a probe's pixels lie in one
// image row).
//
// The forest posterior of pixel (x, y): the leaf of every tree (its index in the
// forest, kept in the CTA's leaf_s, [tree][thread]), then the leaf posteriors summed
// in tree order and divided by the tree count, written planar with stride plane.
// post: rows of K4 float4 (the classes padded to a multiple of four), so that four
// classes of a leaf are one load; the planes are written with the streaming hint
// (they are not read here, and the images and records stay in L2).
template <class P, bool AF = false>
PD_D void predict_pixel(const ImageRef<typename P::img_t> &im, uint32_t x, uint32_t y, bool masked_out, float *o,
                        size_t plane, const Node<P, AF> *__restrict__ nodes, const float4 *__restrict__ post,
                        const TreeMeta *__restrict__ meta, uint32_t n_trees, uint32_t K, int32_t *leaf_s,
                        uint32_t tid) {
  if (masked_out) {
    for (uint32_t l = 0; l < K; l++) o[l * plane] = 0.0f;
    return;
  }
  const Pixel<P, AF> px(im, (int32_t)x, (int32_t)y);
  for (uint32_t t = 0; t < n_trees; t++) {
    const unsigned long long off = meta[t].off;
    leaf_s[t * kPredThreads + tid] = (int32_t)off + walk<P, AF>(px, nodes + off, meta[t].depth);
  }
  const float nt = (float)n_trees;
  const uint32_t K4 = (K + 3) / 4;
  for (uint32_t q = 0; q < K4; q++) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (uint32_t t = 0; t < n_trees; t++) {
      const float4 p = ldg(post + (size_t)(uint32_t)leaf_s[t * kPredThreads + tid] * K4 + q);
      acc[0] = acc[0] + p.x;
      acc[1] = acc[1] + p.y;
      acc[2] = acc[2] + p.z;
      acc[3] = acc[3] + p.w;
    }
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
      if (4 * q + i < K) __stcs(o + (4 * q + i) * plane, fdiv(acc[i], nt));
  }
}

// post [n][K] -> out [n][ceil(K / 4)], padded with zeros: a thread per word of four
// classes.  Runs once per forest, where K is no multiple of four.
static __global__ void k_pad_posteriors(const float *__restrict__ post, unsigned long long n, uint32_t K,
                                        float4 *__restrict__ out) {
  const uint32_t K4 = (K + 3) / 4;
  const unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  if (i >= n * K4) return;
  const unsigned long long node = i >> 32 ? i / K4 : (uint32_t)i / K4;
  const uint32_t l = 4 * (uint32_t)(i - node * K4);
  const float *p = post + node * K + l;
  out[i] = make_float4(p[0], l + 1 < K ? p[1] : 0.0f, l + 2 < K ? p[2] : 0.0f, l + 3 < K ? p[3] : 0.0f);
}

// grid (ceil(W/32), ceil(H/8), n_images); dynamic smem n_trees*256 int32.
template <class P, bool AF = false>
__global__ void __launch_bounds__(kPredThreads) k_predict_posterior(
    const uint8_t *__restrict__ images, uint64_t img_bytes, uint32_t W, uint32_t H,
    const uint8_t *__restrict__ masks, float *__restrict__ out, const Node<P, AF> *__restrict__ nodes,
    const float4 *__restrict__ post, const TreeMeta *__restrict__ meta, uint32_t n_trees, uint32_t K,
    const uint32_t *__restrict__ magic) {
  using ImgT = typename P::img_t;
  extern __shared__ int32_t leaf_s[];
  const uint32_t tid = threadIdx.y * kPredX + threadIdx.x;
  const uint32_t x = blockIdx.x * kPredX + threadIdx.x, y = blockIdx.y * kPredY + threadIdx.y, z = blockIdx.z;
  if (x >= W || y >= H) return;
  const size_t P_ = (size_t)W * H, pix = (size_t)y * W + x;
  ImageRef<ImgT> im;
  im.data = reinterpret_cast<const ImgT *>(images + (size_t)z * img_bytes);
  im.w = (int32_t)W;
  im.h = (int32_t)H;
  im.magic = magic;
  predict_pixel<P, AF>(im, x, y, masks && !masks[(size_t)z * P_ + pix], out + (size_t)z * K * P_ + pix, P_, nodes,
                       post, meta, n_trees, K, leaf_s, tid);
}

// One image of a mixed-size batch: byte offsets of its pixels, mask and
// posterior planes in the batch buffers, its size and its first tile.
struct BatchImage {
  unsigned long long img_off, mask_off, out_off;
  uint32_t w, h, tiles_x, tile0;
  uint32_t has_mask, pad;
};

// A mixed-size batch in one launch: CTA b serves tile b of the concatenated
// tile lists (32x8 pixels; its image found by binary search over tile0).
template <class P, bool AF = false>
__global__ void __launch_bounds__(kPredThreads) k_predict_batch(
    const uint8_t *__restrict__ images, const uint8_t *__restrict__ masks, uint8_t *__restrict__ out,
    const BatchImage *__restrict__ batch, uint32_t n, const Node<P, AF> *__restrict__ nodes,
    const float4 *__restrict__ post, const TreeMeta *__restrict__ meta, uint32_t n_trees, uint32_t K,
    const uint32_t *__restrict__ magic) {
  using ImgT = typename P::img_t;
  extern __shared__ int32_t leaf_s[];
  uint32_t lo = 0, hi = n;  // the last image whose first tile is <= blockIdx.x
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (batch[mid].tile0 <= blockIdx.x) lo = mid;
    else hi = mid;
  }
  const BatchImage b = batch[lo];
  const uint32_t t = blockIdx.x - b.tile0;
  const uint32_t x = (t % b.tiles_x) * kPredX + threadIdx.x, y = (t / b.tiles_x) * kPredY + threadIdx.y;
  if (x >= b.w || y >= b.h) return;
  const uint32_t tid = threadIdx.y * kPredX + threadIdx.x;
  const size_t P_ = (size_t)b.w * b.h, pix = (size_t)y * b.w + x;
  ImageRef<ImgT> im;
  im.data = reinterpret_cast<const ImgT *>(images + b.img_off);
  im.w = (int32_t)b.w;
  im.h = (int32_t)b.h;
  im.magic = magic;
  const bool masked_out = b.has_mask && !masks[b.mask_off + pix];
  predict_pixel<P, AF>(im, x, y, masked_out, reinterpret_cast<float *>(out + b.out_off) + pix, P_, nodes, post, meta,
                       n_trees, K, leaf_s, tid);
}

template <class P, bool AF = false>
__global__ void __launch_bounds__(kPredThreads) k_predict_leaf(const uint8_t *__restrict__ image, uint32_t W,
                                                               uint32_t H, const uint8_t *__restrict__ mask,
                                                               int32_t *__restrict__ out,
                                                               const Node<P, AF> *__restrict__ nodes,
                                                               uint32_t depth, const uint32_t *__restrict__ magic) {
  using ImgT = typename P::img_t;
  const uint32_t x = blockIdx.x * kPredX + threadIdx.x, y = blockIdx.y * kPredY + threadIdx.y;
  if (x >= W || y >= H) return;
  const size_t pix = (size_t)y * W + x;
  if (mask && !mask[pix]) {
    out[pix] = 0;
    return;
  }
  ImageRef<ImgT> im;
  im.data = reinterpret_cast<const ImgT *>(image);
  im.w = (int32_t)W;
  im.h = (int32_t)H;
  im.magic = magic;
  out[pix] = walk<P, AF>(Pixel<P, AF>(im, (int32_t)x, (int32_t)y), nodes, depth);
}

// One step of the per-pixel node map of features that read the tree
// (kernels/predict.cl:36-85, launched once per level by
// cl_tree_trainer_impl_traverse_ts.hpp:215-232 and cl_classifier_impl.hpp:478-520):
// a pixel inside the mask whose node has children moves to the child its
// feature selects -- the feature reading the map before the step and the tree
// as seen from that map's level -- and every other pixel keeps its node.  Pixel q of the concatenated images
// (image i starts at map_off[i]; n_images + 1 offsets).
struct NodeMapStep {
  const uint8_t *pixels;
  const uint64_t *img_off;   // byte offset of each image
  const uint32_t *img_wh;    // w | h << 16
  const uint64_t *map_off;
  uint32_t n_images;
  uint64_t n_pix;
  const uint8_t *mask;       // per pixel (nonzero: inside); null: every pixel
  const int32_t *map_in;
  int32_t *map_out;
  const int32_t *lc;
  const void *feat, *thr;    // feat_t [node][D], [node]
  const float *post;
  uint32_t n_classes;
  int32_t level, n_nodes;    // the level of map_in (root 0), the tree's node count
  const uint32_t *magic;
};

template <class P>
__global__ void __launch_bounds__(256) k_node_map_step(NodeMapStep a) {
  using FeatT = typename P::feat_t;
  using ImgT = typename P::img_t;
  constexpr int D = P::kFeatDim;
  const uint64_t q = (uint64_t)blockIdx.x * 256u + threadIdx.x;
  if (q >= a.n_pix) return;
  const int32_t n = a.map_in[q];
  int32_t out = n;
  const int32_t c = (a.mask && !a.mask[q]) ? -1 : a.lc[n];
  if (c >= 0) {
    uint32_t lo = 0, hi = a.n_images;  // the last image starting at or before q
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (a.map_off[mid] <= q) lo = mid;
      else hi = mid;
    }
    const uint32_t wh = a.img_wh[lo], w = wh & 0xffffu;
    const uint64_t pix = q - a.map_off[lo];
    ImageRef<ImgT> im;
    im.data = reinterpret_cast<const ImgT *>(a.pixels + a.img_off[lo]);
    im.w = (int32_t)w;
    im.h = (int32_t)(wh >> 16);
    im.magic = a.magic;
    im.nodes = a.map_in + a.map_off[lo];
    im.tree_lc = a.lc;
    im.tree_post = a.post;
    im.n_classes = a.n_classes;
    im.tree_level = a.level;
    im.tree_nodes = a.n_nodes;
    const FeatT *fp = static_cast<const FeatT *>(a.feat) + (size_t)n * D;
    FeatT fv[D];
#pragma unroll
    for (int d = 0; d < D; d++) fv[d] = fp[d];
    const auto prep = P::prepare(im, (int32_t)(pix % w), (int32_t)(pix / w));
    const FeatT resp = P::eval(prep, fv);
    out = c + (resp > static_cast<const FeatT *>(a.thr)[n] ? 1 : 0);
  }
  a.map_out[q] = out;
}

}  // namespace pd
