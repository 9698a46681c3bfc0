// Pixel samplers on the GPU: the reference's UniformImageSampler
// (uniform_image_sampler_impl.hpp:34-63) and ClassWeightedImageSampler
// (classweighted_image_sampler_impl.hpp:25-120) over batches of images, with
// the samples the reference's code returns.
//
// Both seed an MT19937 with the CRC-32 of the image bytes XOR the sampler seed,
// so every image is sampled on its own:
//  1. k_sample_scan, over all images at once (HBM-bound): the CRC-32 of each
//     image as the XOR of per-thread checksums of its bytes, each moved to its
//     place by a multiplication modulo the CRC polynomial, and the number of
//     labelled pixels.
//  2. uniform: one CTA per image (k_sample_uniform): MT19937 blocks of 624 words,
//     each twisted in three parallel phases, Boost's bucket method on every draw
//     (accepted draws keep their order by a block scan), a bucket sort of the
//     drawn ranks, one pass over the labels that maps ranks to pixel indices.
//  3. class-weighted: the per-class reservoir in scan order, in parallel over
//     segments of 512 pixels.  A pixel's count within its class and its draw's
//     index depend only on the class counts before it, so
//     - k_class_counts counts every segment's classes, k_class_prefix turns the
//       counts of an image into each segment's counts and first draw;
//     - k_mt_draws writes each image's MT19937 outputs (the one serial chain left);
//     - k_reservoir takes a warp per segment: ranks from ballots, draws by index; a
//       write lands by atomicMax on its slot (pixel order is scan order, so the
//       last writer of the sequential loop wins);
//     - k_bucket_samples gathers and sorts the buckets.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <thread>
#include <vector>

#include "pd_ctx.cuh"

namespace pd {
namespace {

constexpr uint32_t kSmThreads = 256;
constexpr uint32_t kSmWarps = kSmThreads / 32;
constexpr uint32_t kCrcPoly = 0xEDB88320u;  // CRC-32, reflected
constexpr uint32_t kGfOne = 0x80000000u;    // x^0 in the reflected representation
constexpr uint32_t kGfX8 = 0x00800000u;     // x^8
// Checksum layout: a work item is a 256 KiB slice of an image's bytes, counted
// from the image's end; warp w streams the slice's 32 KiB region w as 16
// blocks of 2 KiB; lane l takes the 64 bytes at 64 l of every block, in two
// chains (even and odd blocks) for instruction-level parallelism.
constexpr uint32_t kPiece = 64;                              // bytes per lane per block
constexpr uint32_t kBlock = 32 * kPiece;                     // 2 KiB
constexpr uint32_t kRegionBlocks = 16;
constexpr uint32_t kRegion = kBlock * kRegionBlocks;         // 32 KiB per warp
constexpr uint32_t kSliceBytes = kRegion * kSmWarps;         // 256 KiB per checksum work item
constexpr uint32_t kGap = 2 * kBlock - kPiece;               // from one piece of a chain to its next
constexpr uint32_t kLabVecsPerItem = 16 * kSmThreads;        // 64 KiB of labels per count work item
constexpr uint32_t kMtN = 624;
constexpr uint32_t kNoError = 0xFFFFFFFFu;

// One image of a sampled batch.  Offsets are into the batch's data, label and
// output arrays.
struct SampImage {
  uint64_t data_lo;   // 16-aligned; bytes between data_lo and the image's first byte are zero
  uint64_t data_end;  // 16-aligned end of the image bytes
  uint64_t lab_off;   // 16-aligned; labels padded with zeros to lab_vecs * 16 bytes
  uint64_t out_off;
  uint32_t n_pix;
  uint32_t lab_vecs;
  uint32_t n_slices;  // checksum work items (kSliceBytes each, counted from data_end)
  uint32_t crc0;      // its first checksum work item (checksum items come first)
  uint32_t lab0;      // its first label work item
  uint32_t seg0;      // its first segment (class-weighted: kSeg pixels each)
  uint64_t draw_off;  // its first draw in the group's draws (class-weighted)
};

// ---- arithmetic modulo the CRC-32 polynomial (reflected: bit 31 is x^0) ----
PD_HD uint32_t gf_mul(uint32_t a, uint32_t b) {
  uint32_t p = 0;
  for (int i = 31; i >= 0; i--) {
    p ^= b & (0u - ((a >> i) & 1u));
    b = (b >> 1) ^ (kCrcPoly & (0u - (b & 1u)));
  }
  return p;
}
// x^(8n): the effect of n zero bytes on a CRC register
PD_HD uint32_t gf_x8n(uint64_t n) {
  uint32_t acc = kGfOne, p = kGfX8;
  while (n) {
    if (n & 1) acc = gf_mul(acc, p);
    p = gf_mul(p, p);
    n >>= 1;
  }
  return acc;
}

// ---- MT19937 (Matsumoto and Nishimura 1998) ----
PD_D uint32_t mt_mix(uint32_t a, uint32_t b) {
  const uint32_t y = (a & 0x80000000u) | (b & 0x7FFFFFFFu);
  return (y >> 1) ^ (0x9908B0DFu & (0u - (y & 1u)));
}
PD_D uint32_t mt_temper(uint32_t y) {
  y ^= y >> 11;
  y ^= (y << 7) & 0x9D2C5680u;
  y ^= (y << 15) & 0xEFC60000u;
  return y ^ (y >> 18);
}
// The seeded state (one thread).
PD_D void mt_seed(uint32_t *x, uint32_t s) {
  x[0] = s;
  for (uint32_t i = 1; i < kMtN; i++) x[i] = 1812433253u * (x[i - 1] ^ (x[i - 1] >> 30)) + i;
}
// The next block d from the state s (all threads of the CTA; ends with a
// barrier).  Word i needs s[i], s[i+1] and s[i+397] for i < 227, the new word
// i-227 after that, and the new word 0 as its successor for i = 623.
PD_D void mt_twist(const uint32_t *s, uint32_t *d) {
  const uint32_t t = threadIdx.x;
  if (t < 227) d[t] = s[t + 397] ^ mt_mix(s[t], s[t + 1]);
  __syncthreads();
  if (t < 227) d[t + 227] = d[t] ^ mt_mix(s[t + 227], s[t + 228]);
  __syncthreads();
  if (t < 170) {
    const uint32_t i = t + 454;
    d[i] = d[i - 227] ^ mt_mix(s[i], i == kMtN - 1 ? d[0] : s[i + 1]);
  }
  __syncthreads();
}

// Exclusive scan of one value per thread over the CTA; *total gets the sum.
// All threads call it (two barriers).
PD_D uint32_t block_scan(uint32_t v, uint32_t *warp_tot, uint32_t *total) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  uint32_t before = 0, tot = 0;
#pragma unroll
  for (uint32_t w = 0; w < kSmWarps; w++) {
    const uint32_t c = warp_tot[w];
    before += w < warp ? c : 0;
    tot += c;
  }
  __syncthreads();
  *total = tot;
  return before + x - v;
}

// Ascending bitonic sort of n (a power of two) words in shared memory; the
// caller has synchronised; ends with a barrier.
PD_D void bitonic_sort(uint32_t *a, uint32_t n) {
  for (uint32_t k = 2; k <= n; k <<= 1)
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < n; i += kSmThreads) {
        const uint32_t l = i ^ j;
        if (l > i) {
          const uint32_t x = a[i], y = a[l];
          if ((x > y) == ((i & k) == 0)) {
            a[i] = y;
            a[l] = x;
          }
        }
      }
      __syncthreads();
    }
}

PD_D uint32_t nonzero_bytes(uint4 x) {
  return (__popc(__vcmpne4(x.x, 0)) + __popc(__vcmpne4(x.y, 0)) + __popc(__vcmpne4(x.z, 0)) +
          __popc(__vcmpne4(x.w, 0))) >> 3;
}
// Index of the r-th (from 0) nonzero byte of x (which has more than r).
PD_D uint32_t nth_nonzero(uint4 x, uint32_t r) {
  const uint32_t m[4] = {__vcmpne4(x.x, 0) & 0x01010101u, __vcmpne4(x.y, 0) & 0x01010101u,
                         __vcmpne4(x.z, 0) & 0x01010101u, __vcmpne4(x.w, 0) & 0x01010101u};
  uint32_t w = 0, sel = m[0];
#pragma unroll
  for (uint32_t i = 0; i < 3; i++) {  // the word
    const uint32_t c = __popc(m[i]);
    if (w == i && r >= c) {
      r -= c;
      w = i + 1;
      sel = m[i + 1];
    }
  }
  // byte j of sel * 0x01010101 counts the nonzero bytes up to j: the first that counts r + 1
  const uint32_t hit = __vcmpgtu4(sel * 0x01010101u, r * 0x01010101u);
  return 4 * w + (((uint32_t)__ffs((int)hit) - 1u) >> 3);
}

// x rounded to `bits` significant bits, to nearest, ties to even.
PD_D uint64_t round_sig(uint64_t x, int bits) {
  const int n = 64 - __clzll((long long)x);
  if (n <= bits) return x;
  const int s = n - bits;
  uint64_t q = x >> s;
  const uint64_t rem = x & ((1ull << s) - 1), half = 1ull << (s - 1);
  if (rem > half || (rem == half && (q & 1))) q++;
  return q << s;
}
// roundf((float)(u * c)) with u = v * 2^-32 in double (uniform_01 on MT19937),
// in integers: the exact product v*c rounded to double's 53 bits, then to
// float's 24, then halves away from zero (classweighted_image_sampler_impl.hpp:91).
PD_D uint32_t reservoir_slot(uint32_t v, uint32_t c) {
  const uint64_t p = (uint64_t)v * c;
  if (p < (1ull << 53)) {
    // the double product is exact: one rounding to float, then an exact scaling
    return (uint32_t)roundf(__fmul_rn(__ull2float_rn(p), 0x1p-32f));
  }
  const uint64_t r = round_sig(round_sig(p, 53), 24);
  return (uint32_t)((r + 0x80000000ull) >> 32);
}

// ------------------------------------------------------------------ kernels --
// Shift constants of the checksum, computed once on the host (x^(8n) is the
// effect of n zero bytes): multiplication tables [4][256] for x^(8 kGap) and
// x^(8 kBlock) (a*X is the XOR of the entries of a's four bytes), x^(8 * bytes
// after lane l's piece in its region) for l < 32, x^(8 * bytes after region
// w in its slice) for w < 8, x^(8 kSliceBytes 2^k) for k < 32.
constexpr uint32_t kShiftGap = 0, kShiftBlock = 1024, kShiftLane = 2048, kShiftWarp = 2080, kShiftSlice = 2088,
                   kShiftWords = 2120;

PD_D uint32_t mul_tab(uint32_t a, const uint32_t *M) {
  return M[a & 0xFFu] ^ M[256 + ((a >> 8) & 0xFFu)] ^ M[512 + ((a >> 16) & 0xFFu)] ^ M[768 + (a >> 24)];
}

PD_D void prefetch_l2(const uint8_t *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// 64 bytes into the CRC register r, one table step per byte.
PD_D uint32_t crc_piece(uint32_t r, const uint4 (&q)[4], const uint32_t *T) {
#pragma unroll
  for (uint32_t i = 0; i < 16; i++) {
    const uint4 &x = q[i >> 2];
    r ^= (i & 3) == 0 ? x.x : (i & 3) == 1 ? x.y : (i & 3) == 2 ? x.z : x.w;
#pragma unroll
    for (uint32_t s = 0; s < 4; s++) r = T[(r & 0xFFu) << 5] ^ (r >> 8);
  }
  return r;
}

// Work items: the checksum slices of all images (counted from each image's
// end), then the label chunks of all images; CTAs take the next item from a
// counter.  crc[] starts at each image's initial-value term, count[] and
// *next at zero.
__global__ void __launch_bounds__(kSmThreads, 4) k_sample_scan(const uint8_t *__restrict__ data,
                                                            const uint8_t *__restrict__ labels,
                                                            const SampImage *__restrict__ imgs,
                                                            const uint32_t *__restrict__ item_img, uint32_t n_items,
                                                            uint32_t n_crc_items, const uint32_t *__restrict__ shifts,
                                                            uint32_t *__restrict__ crc, uint32_t *__restrict__ count,
                                                            uint32_t *__restrict__ next) {
  // byte table, one copy per bank: entry e of lane l at [e * 32 + l]
  __shared__ uint32_t tab[256 * 32];
  __shared__ uint32_t mgap[1024], mblock[1024];
  __shared__ uint32_t xs[32];
  __shared__ uint32_t red[kSmWarps];
  __shared__ uint32_t s_item;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  {
    uint32_t r = t;
    for (int k = 0; k < 8; k++) r = (r >> 1) ^ (kCrcPoly & (0u - (r & 1u)));
    for (uint32_t i = 0; i < 32; i++) tab[t * 32 + ((i + lane) & 31)] = r;
  }
  if (t == 0) s_item = atomicAdd(next, 1u);
  for (uint32_t i = t; i < 1024; i += kSmThreads) {
    mgap[i] = shifts[kShiftGap + i];
    mblock[i] = shifts[kShiftBlock + i];
  }
  if (t < 32) xs[t] = shifts[kShiftSlice + t];
  const uint32_t x_lane = shifts[kShiftLane + lane], x_warp = shifts[kShiftWarp + warp];
  __syncthreads();
  const uint32_t *T = tab + lane;
  for (;;) {
    const uint32_t item = s_item;
    if (item >= n_items) break;
    const uint32_t im = item_img[item];
    const SampImage g = imgs[im];
    if (item < n_crc_items) {
      const uint32_t local = item - g.crc0;
      const int64_t r_end = (int64_t)g.data_end - (int64_t)local * kSliceBytes - (int64_t)(kSmWarps - 1 - warp) * kRegion;
      const int64_t r_beg = r_end - kRegion, lo = (int64_t)g.data_lo;
      uint32_t acc = 0;
      if (r_end > lo) {  // warp-uniform: this warp's region holds image bytes
        const uint8_t *rb = data + r_beg;  // only dereferenced at or after data + lo
        // the first blocks into L2 (lanes 0-15: the 16 lines of one block)
        if (lane < 16)
#pragma unroll
          for (uint32_t j = 0; j < 4; j++)
            if (r_beg + (int64_t)(j * kBlock) >= lo) prefetch_l2(rb + j * kBlock + lane * 128);
        uint32_t s0 = 0, s1 = 0;
#pragma unroll 1
        for (uint32_t j = 0; j < kRegionBlocks; j += 2) {
          if (j + 4 < kRegionBlocks) {
            const uint32_t pj = j + 4 + (lane >> 4);
            if (r_beg + (int64_t)(pj * kBlock) >= lo) prefetch_l2(rb + pj * kBlock + (lane & 15) * 128);
          }
          uint4 q0[4], q1[4];
#pragma unroll
          for (uint32_t i = 0; i < 4; i++) {
            const int64_t a0 = r_beg + (int64_t)(j * kBlock + lane * kPiece + i * 16);
            const int64_t a1 = a0 + kBlock;
            q0[i] = a0 >= lo ? __ldg(reinterpret_cast<const uint4 *>(data + a0)) : make_uint4(0, 0, 0, 0);
            q1[i] = a1 >= lo ? __ldg(reinterpret_cast<const uint4 *>(data + a1)) : make_uint4(0, 0, 0, 0);
          }
          s0 = crc_piece(mul_tab(s0, mgap), q0, T);
          s1 = crc_piece(mul_tab(s1, mgap), q1, T);
        }
        // chain 0 ends one block before chain 1; then to the end of the region
        acc = mul_tab(s0, mblock) ^ s1;
        if (acc) acc = gf_mul(acc, x_lane);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc ^= __shfl_xor_sync(0xFFFFFFFFu, acc, o);
      if (lane == 0) red[warp] = acc ? gf_mul(acc, x_warp) : 0u;
      __syncthreads();
      if (t == 0) {
        uint32_t tot = 0;
        for (uint32_t w = 0; w < kSmWarps; w++) tot ^= red[w];
        if (tot) {
          for (uint32_t k = 0; k < 32; k++)
            if ((local >> k) & 1u) tot = gf_mul(tot, xs[k]);
          atomicXor(&crc[im], tot);
        }
      }
    } else {
      const uint32_t v0 = (item - g.lab0) * kLabVecsPerItem;
      const uint4 *L = reinterpret_cast<const uint4 *>(labels + g.lab_off);
      uint32_t n = 0;
#pragma unroll 4
      for (uint32_t i = 0; i < kLabVecsPerItem / kSmThreads; i++) {
        const uint32_t vi = v0 + i * kSmThreads + t;
        if (vi < g.lab_vecs) n += nonzero_bytes(__ldg(L + vi));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xFFFFFFFFu, n, o);
      if (lane == 0) red[warp] = n;
      __syncthreads();
      if (t == 0) {
        uint32_t tot = 0;
        for (uint32_t w = 0; w < kSmWarps; w++) tot += red[w];
        if (tot) atomicAdd(&count[im], tot);
      }
    }
    __syncthreads();  // everyone has read s_item and red[]
    if (t == 0) s_item = atomicAdd(next, 1u);
    __syncthreads();
  }
}

constexpr uint32_t kWalkVecs = 4;  // label vectors (64 pixels) per thread per step of the rank walk

PD_D void walk_load(uint4 (&x)[kWalkVecs], const uint4 *L, uint32_t v, uint32_t n_vecs) {
#pragma unroll
  for (uint32_t i = 0; i < kWalkVecs; i++) x[i] = v + i < n_vecs ? __ldg(L + v + i) : make_uint4(0, 0, 0, 0);
}

// keys[0, n) (values below `range`, spread evenly over it) -> sorted[0, n), by the
// whole CTA: one bucket per key on average (a monotone map of the value), a prefix
// over the bucket counts, and an insertion sort inside each bucket.  cnt: `buckets`
// words (a multiple of kSmThreads).  A bitonic sort of 2048 keys takes 66 barriers,
// this nine.  Ends with a barrier.
PD_D void bucket_sort(const uint32_t *keys, uint32_t n, uint32_t range, uint32_t *cnt, uint32_t buckets,
                      uint32_t *sorted, uint32_t *wtot) {
  const uint32_t t = threadIdx.x, per = buckets / kSmThreads;
  const double scale = (double)buckets / (double)range;
  auto bucket_of = [&](uint32_t q) { return min(buckets - 1u, (uint32_t)((double)q * scale)); };
  for (uint32_t i = t; i < buckets; i += kSmThreads) cnt[i] = 0u;
  __syncthreads();
  for (uint32_t i = t; i < n; i += kSmThreads) atomicAdd(&cnt[bucket_of(keys[i])], 1u);
  __syncthreads();
  uint32_t sum = 0, total;
  for (uint32_t i = 0; i < per; i++) sum += cnt[t * per + i];
  uint32_t run = block_scan(sum, wtot, &total);
  const uint32_t beg = run;
  for (uint32_t i = 0; i < per; i++) {  // first position of each bucket
    const uint32_t c = cnt[t * per + i];
    cnt[t * per + i] = run;
    run += c;
  }
  __syncthreads();
  for (uint32_t i = t; i < n; i += kSmThreads) {
    const uint32_t q = keys[i];
    sorted[atomicAdd(&cnt[bucket_of(q)], 1u)] = q;  // cnt: the bucket's end when all are in
  }
  __syncthreads();
  uint32_t b = beg;
  for (uint32_t i = 0; i < per; i++) {
    const uint32_t e = cnt[t * per + i];
    for (uint32_t x = b + 1; x < e; x++) {
      const uint32_t q = sorted[x];
      uint32_t y = x;
      for (; y > b && sorted[y - 1] > q; y--) sorted[y] = sorted[y - 1];
      sorted[y] = q;
    }
    b = e;
  }
  __syncthreads();
}

// UniformImageSampler::sample, one CTA per image.  Dynamic shared memory: the draws
// and the sorted draws (n_samples words each), then `buckets` words.
// Latency-bound (barriers, the seed's serial chain).  500 maps of 640x480, 2000 samples:
// 0.077 ms; with a bitonic sort, and a walk in which every thread searched the keys
// and stepped through bytes at every step, 0.140.
__global__ void __launch_bounds__(kSmThreads) k_sample_uniform(const uint8_t *__restrict__ labels,
                                                               const SampImage *__restrict__ imgs,
                                                               const uint32_t *__restrict__ crc,
                                                               const uint32_t *__restrict__ count, uint32_t n_samples,
                                                               uint32_t seed, uint32_t buckets,
                                                               uint32_t *__restrict__ out,
                                                               uint32_t *__restrict__ out_count,
                                                               uint32_t *__restrict__ err) {
  extern __shared__ uint32_t dyn[];
  uint32_t *drawn = dyn, *keys = dyn + n_samples, *cnt = keys + n_samples;
  __shared__ uint32_t mt[2][kMtN];
  __shared__ uint32_t wtot[kSmWarps];
  __shared__ uint32_t s_base[kSmThreads + 1], s_vec[kSmThreads];
  const uint32_t im = blockIdx.x, t = threadIdx.x;
  const SampImage g = imgs[im];
  const uint32_t n = count[im];
  if (n == 0) {  // no labelled pixel (the reference draws from an empty buffer)
    if (t == 0) out_count[im] = 0;
    return;
  }
  if (n == 1) {  // range 0: Boost returns the lower bound without drawing
    for (uint32_t i = t; i < n_samples; i += kSmThreads) keys[i] = 0;
    __syncthreads();
  } else {
    if (t == 0) mt_seed(mt[0], crc[im] ^ seed);
    __syncthreads();
    const uint32_t bucket = (uint32_t)(0x100000000ull / n);
    // a draw is accepted with probability above 1/2: twice the blocks that
    // takes on average, and 64 more, end the loop in any case
    const uint32_t max_blocks = 4 * n_samples / kMtN + 64;
    uint32_t got = 0, cur = 0, blocks = 0;
    while (got < n_samples) {
      if (blocks++ == max_blocks) {
        if (t == 0) atomicMin(err + 1, im);
        for (uint32_t i = got + t; i < n_samples; i += kSmThreads) drawn[i] = 0;  // the call fails
        break;
      }
      mt_twist(mt[cur], mt[cur ^ 1]);
      cur ^= 1;
      uint32_t q[3] = {n, n, n}, ok = 0;
      if (t < kMtN / 3) {
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) {
          q[k] = mt_temper(mt[cur][3 * t + k]) / bucket;
          ok += q[k] < n;
        }
      }
      uint32_t total;
      uint32_t pos = got + block_scan(ok, wtot, &total);
#pragma unroll
      for (uint32_t k = 0; k < 3; k++)
        if (q[k] < n) {
          if (pos < n_samples) drawn[pos] = q[k];
          pos++;
        }
      got += total;
    }
    __syncthreads();
    bucket_sort(drawn, n_samples, n, cnt, buckets, keys, wtot);
  }
  // ranks among the labelled pixels -> pixel indices, in one pass over the labels:
  // kWalkVecs label vectors per thread per step, the next step's loaded ahead; then a
  // thread per sample of the step finds the thread whose pixels hold its rank, the
  // vector and the byte
  const uint4 *L = reinterpret_cast<const uint4 *>(labels + g.lab_off);
  const uint32_t last = keys[n_samples - 1];
  uint32_t *o = out + g.out_off;
  uint32_t run = 0, done = 0;  // labelled pixels and samples before the step
  uint4 xa[kWalkVecs], xb[kWalkVecs];
  walk_load(xa, L, t * kWalkVecs, g.lab_vecs);
  for (uint32_t v0 = 0; v0 < g.lab_vecs && run <= last; v0 += kSmThreads * kWalkVecs) {
    walk_load(xb, L, v0 + kSmThreads * kWalkVecs + t * kWalkVecs, g.lab_vecs);
    uint32_t ct = 0, vec = 0;  // vec: labelled pixels before vectors 1, 2, 3 of the thread (a byte each)
#pragma unroll
    for (uint32_t i = 0; i < kWalkVecs; i++) {
      vec |= ct << (8 * i);
      ct += nonzero_bytes(xa[i]);
    }
    uint32_t total;
    s_base[t] = run + block_scan(ct, wtot, &total);
    s_vec[t] = vec;
    if (t == 0) s_base[kSmThreads] = run + total;
    __syncthreads();
    const uint32_t end = run + total;
    for (;;) {  // kSmThreads samples at a time (uniform: every thread sees the same bounds)
      const uint32_t i = done + t;
      const uint32_t key = i < n_samples ? keys[i] : 0xFFFFFFFFu;
      if (key < end) {
        uint32_t lo = 0, hi = kSmThreads;  // the last thread whose base is at or below the key
#pragma unroll
        for (uint32_t s = 0; s < 8; s++) {
          const uint32_t mid = (lo + hi) >> 1;
          if (s_base[mid] <= key) lo = mid;
          else hi = mid;
        }
        uint32_t r = key - s_base[lo];
        const uint32_t pv = s_vec[lo];
        uint32_t k = 0;
#pragma unroll
        for (uint32_t j = 1; j < kWalkVecs; j++) k += r >= ((pv >> (8 * j)) & 0xFFu) ? 1u : 0u;
        r -= (pv >> (8 * k)) & 0xFFu;
        const uint32_t v = v0 + lo * kWalkVecs + k;
        o[i] = v * 16 + nth_nonzero(__ldg(L + v), r);
      }
      const uint32_t taken = (uint32_t)__syncthreads_count(key < end);
      done += taken;
      if (taken < kSmThreads) break;
    }
    run = end;
#pragma unroll
    for (uint32_t i = 0; i < kWalkVecs; i++) xa[i] = xb[i];
  }
  if (t == 0) out_count[im] = n_samples;
}

// ---- ClassWeightedImageSampler::sample ----
// 500 maps of 640x480, 2000 samples, 9 classes: one CTA walking each image in
// 1024-pixel steps (three barriers per 624 draws, four per step) took 1.07 ms.  The
// kernels below take 0.09 (counts), 0.02 (prefix), 0.20 (draws), 0.38 (reservoir) and
// 0.02 ms (samples), and the checksum scan no longer reads the labels (0.129 -> 0.119).
constexpr uint32_t kSeg = 512;  // pixels of a segment (16 per lane of a warp)
constexpr uint32_t kSegRun = 2;    // segments of a k_reservoir warp, one after the other
constexpr uint32_t kSegGroup = 4;  // its rows of 32 pixels in flight together
constexpr int kResCtas = 5;

// Class counts of every segment: class k of segment s of an image at
// counts[seg0 * n_classes + k * segs + s].  A warp per segment; 32 classes at a time
// in counters of the lane's own ([class][lane], no conflicts): one shared add per
// label, then a warp sum per class.  Labels above n_classes are errors (err: the
// lowest image).  Issue-bound (300 maps, 92 MB of labels: 59 us, 86 % issue-active).
// Grid: (segments of the largest image / kSmWarps, images).
__global__ void __launch_bounds__(kSmThreads) k_class_counts(const uint8_t *__restrict__ labels,
                                                             const SampImage *__restrict__ imgs, uint32_t first,
                                                             uint32_t n_classes, uint32_t *__restrict__ counts,
                                                             uint32_t *__restrict__ err) {
  extern __shared__ uint32_t cnt_all[];  // [warps][min(n_classes, 32) + 1][32]; row 0: every other label
  const uint32_t rows = min(n_classes, 32u) + 1;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, im = first + blockIdx.y;
  uint32_t *mine = cnt_all + warp * rows * 32 + lane;
  const SampImage g = imgs[im];
  const uint32_t s = blockIdx.x * kSmWarps + warp, segs = (g.n_pix + kSeg - 1) / kSeg;
  if (s >= segs) return;
  // 16 labels a lane (zeros past the image), in any order
  const uint32_t p = s * kSeg + 16 * lane;
  const uint4 q = p < g.lab_vecs * 16u ? __ldg(reinterpret_cast<const uint4 *>(labels + g.lab_off + p)) : make_uint4(0, 0, 0, 0);
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  if (!__any_sync(0xFFFFFFFFu, (q.x | q.y | q.z | q.w) != 0u)) {  // a segment without labels
    for (uint32_t k = lane; k < n_classes; k += 32) counts[(size_t)g.seg0 * n_classes + (size_t)k * segs + s] = 0u;
    return;
  }
  uint32_t bad = 0;
  for (uint32_t k0 = 0; k0 < n_classes; k0 += 32) {
    const uint32_t nk = min(n_classes - k0, 32u);
    for (uint32_t k = 0; k <= nk; k++) mine[k * 32] = 0u;
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) {
      const uint32_t l = (w[i >> 2] >> (8 * (i & 3))) & 0xFFu, k = l - k0;
      bad |= l > n_classes;
      atomicAdd(&mine[(k <= nk ? k : 0u) * 32], 1u);  // the lane's own word: no wait between the adds
    }
    uint32_t out = 0;  // lane k: class k0 + k
    for (uint32_t k = 0; k < nk; k++) {
      const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, mine[(k + 1) * 32]);
      if (lane == k) out = sum;
    }
    if (lane < nk) counts[(size_t)g.seg0 * n_classes + (size_t)(k0 + lane) * segs + s] = out;
  }
  if (__any_sync(0xFFFFFFFFu, bad) && lane == 0) atomicMin(err, im);
}

// counts of an image's segments -> the pixels of each class before the segment (in
// place), the class totals, and the index of each segment's first draw: a pixel
// draws when its class's bucket is full.  One CTA per image, a warp per class; it also
// empties the image's slots.
__global__ void __launch_bounds__(kSmThreads) k_class_prefix(const SampImage *__restrict__ imgs, uint32_t n_classes,
                                                             const uint32_t *__restrict__ bucket_size,
                                                             uint32_t *__restrict__ counts, uint32_t *__restrict__ draw0,
                                                             uint32_t *__restrict__ class_tot,
                                                             uint32_t *__restrict__ n_draws,
                                                             uint32_t *__restrict__ slots, uint32_t stride) {
  for (uint32_t i = threadIdx.x; i < stride; i += kSmThreads) slots[(size_t)blockIdx.x * stride + i] = 0u;
  const SampImage g = imgs[blockIdx.x];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t segs = (g.n_pix + kSeg - 1) / kSeg;
  uint32_t *c = counts + (size_t)g.seg0 * n_classes;
  for (uint32_t k = warp; k < n_classes; k += kSmWarps) {
    uint32_t *ck = c + (size_t)k * segs, run = 0;
    uint32_t nxt = lane < segs ? ck[lane] : 0u;
    for (uint32_t s0 = 0; s0 < segs; s0 += 32) {
      const uint32_t s = s0 + lane, v = nxt;
      nxt = s + 32 < segs ? ck[s + 32] : 0u;  // the next step's, ahead
      uint32_t x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      if (s < segs) ck[s] = run + x - v;
      run += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    if (lane == 0) class_tot[(size_t)blockIdx.x * n_classes + k] = run;
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s <= segs; s += kSmThreads) {
    uint32_t d = 0;
#pragma unroll 8
    for (uint32_t k = 0; k < n_classes; k++) {
      const uint32_t seen = s < segs ? c[(size_t)k * segs + s] : class_tot[(size_t)blockIdx.x * n_classes + k];
      d += seen > bucket_size[k] ? seen - bucket_size[k] : 0u;
    }
    if (s < segs) draw0[g.seg0 + s] = d;
    else n_draws[blockIdx.x] = d;
  }
}

// The first n_draws MT19937 outputs of every image of a group, at draws + g.draw_off.
// One CTA of 112 threads per image: word n + 624 needs words n, n + 1 and n + 397, so
// 224 words go at a time, two a thread (64-bit shared accesses), one barrier each; the
// words run through a linear array (fixed offsets from one pointer) whose last 624
// move to its start at the end of a lap.  A step's words are tempered and stored
// while the next step's loads are in flight, off the chain.  Bound by the chain's
// latency (300 images, two an SM: 48 % issue-active, ALU pipe 50 %, 301 MB written in
// 0.15 ms); one word a thread in 8 warps 0.22 ms for 500 images, four in 2 warps 0.21,
// this 0.20.  Every thread of the CTA works in every step: the barriers see whole warps.
constexpr uint32_t kMtStep = 224, kMtThreads = kMtStep / 2, kMtLap = 15;
constexpr uint32_t kMtWords = kMtN + kMtLap * kMtStep;
__global__ void __launch_bounds__(kMtThreads) k_mt_draws(const SampImage *__restrict__ imgs, uint32_t first,
                                                         const uint32_t *__restrict__ crc, uint32_t seed,
                                                         const uint32_t *__restrict__ n_draws,
                                                         uint32_t *__restrict__ draws) {
  __shared__ __align__(16) uint32_t x[kMtWords];
  const uint32_t im = first + blockIdx.x, t = threadIdx.x, n = n_draws[im];
  if (n == 0) return;
  uint32_t *out = draws + imgs[im].draw_off + 2 * t;  // 8-byte aligned; whole pairs are kept
  if (t == 0) mt_seed(x, crc[im] ^ seed);
  __syncthreads();
  uint2 v = make_uint2(0, 0);
  for (uint32_t d0 = 0; d0 < n;) {
    uint32_t *p = x + 2 * t;
    for (uint32_t lap = 0; lap < kMtLap && d0 < n; lap++, d0 += kMtStep, p += kMtStep) {
      const uint2 a = *reinterpret_cast<const uint2 *>(p), b = *reinterpret_cast<const uint2 *>(p + 396),
                  c = *reinterpret_cast<const uint2 *>(p + 398);
      const uint32_t a2 = p[2];
      if (d0) {  // the step before: draws d0 - kMtStep + 2 t (all below n: n > d0)
        *reinterpret_cast<uint2 *>(out) = make_uint2(mt_temper(v.x), mt_temper(v.y));
        out += kMtStep;
      }
      v = make_uint2(b.y ^ mt_mix(a.x, a.y), c.x ^ mt_mix(a.y, a2));
      *reinterpret_cast<uint2 *>(p + kMtN) = v;
      __syncthreads();
    }
    if (d0 >= n) break;
    for (uint32_t i = t; i < kMtN; i += kMtThreads) x[i] = x[kMtLap * kMtStep + i];  // the two ranges are apart
    __syncthreads();
  }
  // the last step: its draws below n
  const uint32_t i = (n - 1) / kMtStep * kMtStep + 2 * t;
  if (i < n) *reinterpret_cast<uint2 *>(out) = make_uint2(mt_temper(v.x), mt_temper(v.y));
}
static_assert(kMtLap * kMtStep >= kMtN, "a lap's end does not overlap its start");

// The reservoir, a warp per kSegRun segments (grid as k_class_counts).  Pixel p of
// class k with c pixels of its class before it takes slot c while the bucket has
// room; else its draw v picks slot roundf(v 2^-32 c), which counts if it lies in the
// bucket.  c and the draw's index come from the segment's prefix and the ballots of
// the rows before it.  floor(v c 2^-32) >= the bucket's size settles nearly every
// draw (the rounding is monotone, and the size a float).
// BITS: of a label, n_classes < 2^BITS; up to 32 classes are counted a lane each (a
// row's mask of class k is lane k's, and goes to the pixels of class k by a shuffle);
// BITS = 8: more classes, counted in shared memory.
// Issue- and ALU-bound (300 maps: 68 instructions per row of 32 pixels, 71 %
// issue-active, ALU pipe 73 %, 36 warps an SM).  500 maps: eight rows in flight with
// four CTAs 0.386 ms, four rows with five 0.378; all rows of a segment unrolled
// 0.48-0.74 (instruction cache).
template <int BITS>
__global__ void __launch_bounds__(kSmThreads, kResCtas) k_reservoir(const uint8_t *__restrict__ labels,
                                                          const SampImage *__restrict__ imgs, uint32_t first,
                                                          uint32_t n_classes,
                                                          const uint32_t *__restrict__ bucket_size,
                                                          const uint32_t *__restrict__ bucket_off,
                                                          const uint32_t *__restrict__ counts,
                                                          const uint32_t *__restrict__ draw0,
                                                          const uint32_t *__restrict__ draws, uint32_t stride,
                                                          uint32_t *__restrict__ slots) {
  constexpr bool WIDE = BITS == 8;
  __shared__ uint32_t s_cnt[WIDE ? kSmWarps : 1][WIDE ? 256 : 1];  // by label
  __shared__ uint32_t bsz[257], boff[257];  // by label; label 0 never fills its bucket
  for (uint32_t k = threadIdx.x; k <= n_classes; k += kSmThreads) {
    bsz[k] = k ? bucket_size[k - 1] : 0xFFFFFFFFu;
    boff[k] = k ? bucket_off[k - 1] : 0u;
  }
  __syncthreads();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  const uint32_t im = first + blockIdx.y;
  const SampImage g = imgs[im];
  const uint32_t segs = (g.n_pix + kSeg - 1) / kSeg;
  const uint32_t s_beg = (blockIdx.x * kSmWarps + warp) * kSegRun, s_end = min(segs, s_beg + kSegRun);
  if (s_beg >= segs) return;
  const uint8_t *lp = labels + g.lab_off;
  // groups of kSegGroup rows of 32 pixels (row i: pixels p + 32 i + lane), the next
  // group's labels loaded ahead; the loop over them stays a loop (unrolled, it
  // outgrows the instruction cache)
  const uint32_t p_beg = s_beg * kSeg, p_end = min(g.n_pix, s_end * kSeg);
  uint32_t nxt[kSegGroup];
  auto load_rows = [&](uint32_t p0) {
#pragma unroll
    for (uint32_t i = 0; i < kSegGroup; i++) {
      const uint32_t p = p0 + 32 * i + lane;
      nxt[i] = p < p_end ? (uint32_t)__ldg(lp + p) : 0u;
    }
  };
  load_rows(p_beg);
  const uint32_t *c0 = counts + (size_t)g.seg0 * n_classes + s_beg;
  uint32_t cnt = 0, flip[BITS];  // lane k: pixels of class k so far; the inverted bits of label k + 1
#pragma unroll
  for (int b = 0; b < BITS; b++) flip[b] = ((lane + 1u) >> b) & 1u ? 0u : 0xFFFFFFFFu;
  if constexpr (WIDE) {
    for (uint32_t l = lane; l <= n_classes; l += 32) s_cnt[warp][l] = l ? c0[(size_t)(l - 1) * segs] : 0u;
    __syncwarp();
  } else {
    cnt = lane < n_classes ? c0[(size_t)lane * segs] : 0u;
  }
  const uint32_t *dr = draws + g.draw_off + draw0[g.seg0 + s_beg];
  uint32_t *sl = slots + (size_t)im * stride;
  // The few pixels that may take a slot queue up, and are settled 32 at a time.
  __shared__ __align__(16) uint4 s_q[kSmWarps][64];  // label, rank, draw, pixel + 1
  uint4 *q = s_q[warp];
  uint32_t nq = 0;
  auto take = [&](uint32_t count) {
    if (lane < count) {
      const uint4 e = q[lane];
      const uint32_t size = bsz[e.x], slot = e.y < size ? e.y : reservoir_slot(e.z, e.y);
      if (slot < size) atomicMax(&sl[boff[e.x] + slot], e.w);
    }
  };
#pragma unroll 1
  for (uint32_t p0 = p_beg; p0 < p_end; p0 += 32 * kSegGroup) {
    uint32_t rows[kSegGroup], rank[kSegGroup], v[kSegGroup];
#pragma unroll
    for (uint32_t i = 0; i < kSegGroup; i++) rows[i] = nxt[i] <= n_classes ? nxt[i] : 0u;  // a larger label is an error
    load_rows(p0 + 32 * kSegGroup);
    // ranks and draws, the draws loaded together
#pragma unroll
    for (uint32_t i = 0; i < kSegGroup; i++) {
      const uint32_t lab = rows[i];
      uint32_t c;
      if constexpr (WIDE) {
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, lab);
        c = s_cnt[warp][lab] + __popc(peers & lt);
        __syncwarp();
        if ((peers & lt) == 0u) s_cnt[warp][lab] += __popc(peers);
        __syncwarp();
      } else {
        uint32_t row = 0xFFFFFFFFu;  // lane k: the row's pixels of class k
#pragma unroll
        for (int b = 0; b < BITS; b++) row &= __ballot_sync(0xFFFFFFFFu, lab & (1u << b)) ^ flip[b];
        c = __shfl_sync(0xFFFFFFFFu, cnt, lab - 1u) + __popc(__shfl_sync(0xFFFFFFFFu, row, lab - 1u) & lt);
        cnt += __popc(row);
      }
      const bool draw = c >= bsz[lab];
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, draw);
      rank[i] = c;
      v[i] = draw ? __ldg(dr + __popc(m & lt)) : 0u;  // 0: takes slot c
      dr += __popc(m);
    }
#pragma unroll
    for (uint32_t i = 0; i < kSegGroup; i++) {
      const uint32_t lab = rows[i];
      const bool may = lab != 0u && __umulhi(v[i], rank[i]) < bsz[lab];
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, may);
      if (m == 0u) continue;
      if (may) q[nq + __popc(m & lt)] = make_uint4(lab, rank[i], v[i], p0 + 32 * i + lane + 1);
      nq += __popc(m);
      if (nq >= 32) {
        __syncwarp();
        take(32);
        nq -= 32;
        const uint4 e = q[32 + lane];  // the rest moves down
        __syncwarp();
        if (lane < nq) q[lane] = e;
        __syncwarp();
      }
    }
  }
  __syncwarp();
  take(nq);
}

// The filled slots of an image, sorted (its samples), one CTA per image.  A pixel
// fills at most one slot, so images of up to kBitmapPixels are sorted by a bitmap in
// shared memory (set the pixels' bits, list them in order); larger ones by the
// bitonic sort.  Dynamic shared memory: the bitmap, or sort_n words.
constexpr uint32_t kBitmapPixels = 1u << 20;  // 128 KB
template <bool BITMAP>
__global__ void __launch_bounds__(kSmThreads) k_bucket_samples(const SampImage *__restrict__ imgs,
                                                               const uint32_t *__restrict__ bucket_size,
                                                               const uint32_t *__restrict__ class_tot,
                                                               uint32_t n_classes, const uint32_t *__restrict__ slots,
                                                               uint32_t stride, uint32_t sort_n,
                                                               uint32_t *__restrict__ out,
                                                               uint32_t *__restrict__ out_count) {
  extern __shared__ __align__(16) uint32_t keys[];
  __shared__ uint32_t wtot[kSmWarps];
  const uint32_t im = blockIdx.x, t = threadIdx.x;
  const SampImage g = imgs[im];
  const uint32_t *sl = slots + (size_t)im * stride;
  uint32_t *o = out + g.out_off;
  if constexpr (BITMAP) {
    const uint32_t words = (g.n_pix + 31) / 32, per = ((words + kSmThreads - 1) / kSmThreads + 3) / 4 * 4;
    for (uint32_t i = t; i < (words + 3) / 4; i += kSmThreads) reinterpret_cast<uint4 *>(keys)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    for (uint32_t i = t; i < stride; i += kSmThreads) {
      const uint32_t p = sl[i] - 1u;  // an empty slot holds 0
      if (p < g.n_pix) atomicOr(&keys[p >> 5], 1u << (p & 31));
    }
    __syncthreads();
    const uint32_t b = min(words, t * per), e = min(words, b + per);
    uint32_t mine = 0, total;
    for (uint32_t i = b; i < e; i++) mine += __popc(keys[i]);
    uint32_t pos = block_scan(mine, wtot, &total);
    for (uint32_t i = b; i < e; i++)
      for (uint32_t m = keys[i]; m; m &= m - 1) o[pos++] = 32 * i + (uint32_t)__ffs((int)m) - 1;
    if (t == 0) out_count[im] = total;
  } else {
    uint32_t mine = 0, total;
    for (uint32_t k = t; k < n_classes; k += kSmThreads)
      mine += min(class_tot[(size_t)im * n_classes + k], bucket_size[k]);
    block_scan(mine, wtot, &total);
    for (uint32_t i = t; i < sort_n; i += kSmThreads) keys[i] = (i < stride ? sl[i] : 0u) - 1u;  // empty: last
    __syncthreads();
    bitonic_sort(keys, sort_n);
    for (uint32_t i = t; i < total; i += kSmThreads) o[i] = keys[i];
    if (t == 0) out_count[im] = total;
  }
}

// ------------------------------------------------------------------- host ----
struct SamplerPlan {
  std::vector<uint32_t> bucket;  // class-weighted bucket sizes
  uint32_t stride = 0, sort_n = 1;
};

int plan_sampler(const pd_sampler *s, SamplerPlan *pl) {
  PD_CHECK(s, PD_ERR_INVALID, "null sampler");
  PD_CHECK(s->kind == PD_SAMPLER_UNIFORM || s->kind == PD_SAMPLER_CLASS_WEIGHTED, PD_ERR_INVALID,
           "unknown sampler kind %d", s->kind);
  PD_CHECK(s->n_samples >= 1, PD_ERR_INVALID, "nSamples must be at least 1");
  PD_CHECK(s->pixel_bytes >= 1, PD_ERR_INVALID, "pixel_bytes must be at least 1");
  uint64_t stride = s->n_samples;
  if (s->kind == PD_SAMPLER_CLASS_WEIGHTED) {
    PD_CHECK(s->n_classes >= 1 && s->n_classes <= 255, PD_ERR_INVALID, "nClasses %u outside [1,255]", s->n_classes);
    // m_perClassBucketSize (classweighted_image_sampler_impl.hpp:33,43): float product, then ceil
    const float p = 1.f / (float)s->n_classes;
    pl->bucket.resize(s->n_classes);
    stride = 0;
    for (uint32_t k = 0; k < s->n_classes; k++) {
      const float w = s->weights ? s->weights[k] : p;
      PD_CHECK(std::isfinite(w) && w >= 0.f, PD_ERR_INVALID, "weight %u is %g (weights must be finite and >= 0)", k,
               (double)w);
      const float b = std::ceil(w * (float)s->n_samples);
      PD_CHECK(b <= (float)PD_SAMPLER_MAX_STRIDE, PD_ERR_UNSUPPORTED, "bucket %u holds %g samples (max %d)", k,
               (double)b, PD_SAMPLER_MAX_STRIDE);
      pl->bucket[k] = (uint32_t)b;
      stride += pl->bucket[k];
    }
  }
  PD_CHECK(stride <= PD_SAMPLER_MAX_STRIDE, PD_ERR_UNSUPPORTED, "%llu samples per image (max %d)",
           (unsigned long long)stride, PD_SAMPLER_MAX_STRIDE);
  pl->stride = (uint32_t)stride;
  pl->sort_n = 1;
  while (pl->sort_n < pl->stride) pl->sort_n <<= 1;
  return PD_OK;
}


// Descriptors, item map, initial checksum terms, zero counts, the error word
// and the class-weighted bucket sizes, in one pinned block uploaded with one
// copy.
struct DescLayout {
  size_t shifts = 0, imgs = 0, items = 0, crc = 0, count = 0, err = 0, bucket = 0, bytes = 0;
  uint32_t n_items = 0, n_crc_items = 0;
  DescLayout() = default;
  DescLayout(uint32_t n, uint32_t n_items, uint32_t n_classes) {
    imgs = shifts + ((4ull * kShiftWords + 15) / 16 * 16);
    items = imgs + sizeof(SampImage) * n;
    crc = items + 4ull * n_items;
    count = crc + 4ull * n;
    err = count + 4ull * n;
    bucket = err + 16;  // err[0], err[1]: errors; err[2]: the scan's work counter
    bytes = bucket + 8ull * n_classes;  // sizes, then offsets
    this->n_items = n_items;
  }
};

// The checksum's shift constants (kShift*), computed once.
const uint32_t *shift_constants() {
  static const std::vector<uint32_t> tab = [] {
    std::vector<uint32_t> v(kShiftWords);
    const uint32_t xg = gf_x8n(kGap), xb = gf_x8n(kBlock);
    for (uint32_t i = 0; i < 4; i++)
      for (uint32_t e = 0; e < 256; e++) {
        v[kShiftGap + i * 256 + e] = gf_mul(e << (8 * i), xg);
        v[kShiftBlock + i * 256 + e] = gf_mul(e << (8 * i), xb);
      }
    for (uint32_t l = 0; l < 32; l++) v[kShiftLane + l] = gf_x8n((uint64_t)kPiece * (31 - l));
    for (uint32_t w = 0; w < kSmWarps; w++) v[kShiftWarp + w] = gf_x8n((uint64_t)kRegion * (kSmWarps - 1 - w));
    uint32_t p = gf_x8n(kSliceBytes);
    for (uint32_t k = 0; k < 32; k++) {
      v[kShiftSlice + k] = p;
      p = gf_mul(p, p);
    }
    return v;
  }();
  return tab.data();
}

// Places of the images' draws in the class-weighted sampler's buffer of MT19937 outputs,
// a word a pixel, for a group of images at a time: a group holds at most `group` words,
// one image at least.  Returns the words that the largest needs.
uint64_t place_draws(SampImage *im, uint32_t n, uint64_t group) {
  uint64_t at = 0, most = 0;
  for (uint32_t i = 0; i < n; i++) {
    const uint64_t words = ((uint64_t)im[i].n_pix + 3) / 4 * 4;
    if (at && at + words > group) at = 0;
    im[i].draw_off = at;
    at += words;
    most = std::max(most, at);
  }
  return most;
}

// That buffer, for images placed in groups of draw_group(ctx): twice the bytes that a
// host batch stages at once (1 GiB, 873 maps of 640x480).  A group should fill the GPU,
// as its draws are a serial chain: the drawing phase of 500 maps in one group takes 0.72
// ms, in two 0.80, in four 1.02, in eight 1.52.  Where that much memory is not free the
// images are placed again in smaller groups; *again: the descriptors changed.
uint64_t draw_group(const pd_ctx *ctx) { return ctx->sample_group / 2; }
int reserve_draws(pd_ctx *ctx, SampImage *im, uint32_t n, bool *again) {
  *again = false;
  uint64_t one = 0, most = 0;
  for (uint32_t i = 0; i < n; i++) {
    const uint64_t words = ((uint64_t)im[i].n_pix + 3) / 4 * 4;
    one = std::max(one, words);
    most = std::max(most, im[i].draw_off + words);
  }
  int rc;
  while ((rc = ctx->sm_draws.ensure(most * 4)) == PD_ERR_NOMEM && most > one) {
    if (!*again) PD_CUDA(cudaStreamSynchronize(ctx->stream));  // the descriptors' upload reads them
    *again = true;
    most = place_draws(im, n, most / 2);
  }
  return rc;
}

// Gives back what a single larger image took of it.
void trim_draws(pd_ctx *ctx) {
  if (ctx->sm_draws.cap > 2 * ctx->sample_group) ctx->sm_draws.release();
}

// The class-weighted sampler's kernels on a batch (images and checksums in place).
// Its scratch -- segment counts, draws, slots -- belongs to the context, like its
// stream: calls on one context are serialised.
int launch_class_weighted(pd_ctx *ctx, const pd_sampler *s, const SamplerPlan &pl, uint32_t n, uint8_t *host_desc,
                          const DescLayout &lay, const uint8_t *labels, SampImage *imgs, const uint32_t *crc,
                          const uint32_t *bucket, uint32_t *out, uint32_t *counts, uint32_t *err, uint64_t *launched) {
  cudaStream_t st = ctx->stream;
  const uint32_t K = s->n_classes;
  SampImage *h = reinterpret_cast<SampImage *>(host_desc + lay.imgs);
  auto segs_of = [&](uint32_t i) { return (h[i].n_pix + kSeg - 1) / kSeg; };
  const uint32_t segs = h[n - 1].seg0 + segs_of(n - 1);
  const size_t slot_bytes = (size_t)n * std::max(1u, pl.stride) * 4;
  bool again = false;
  PD_TRY(reserve_draws(ctx, h, n, &again));
  if (again) PD_CUDA(h2d(ctx, imgs, h, sizeof(SampImage) * n));
  PD_TRY(ctx->sm_counts.ensure(((size_t)segs * (K + 1) + (size_t)n * (K + 1)) * 4));
  PD_TRY(ctx->sm_slots.ensure(slot_bytes));
  uint32_t *c = ctx->sm_counts.as<uint32_t>(), *draw0 = c + (size_t)segs * K, *tot = draw0 + segs,
           *n_draws = tot + (size_t)n * K, *draws = ctx->sm_draws.as<uint32_t>(), *slots = ctx->sm_slots.as<uint32_t>();
  const uint32_t *bsz = bucket, *boff = bucket + K;
  *launched = 2;
  // CTAs of images [first, last): the segments of the largest, up to 65535 images a grid
  auto grid_of = [&](uint32_t first, uint32_t last, uint32_t per_warp) {
    uint32_t most = 0;
    for (uint32_t i = first; i < last; i++) most = std::max(most, segs_of(i));
    return dim3((most + kSmWarps * per_warp - 1) / (kSmWarps * per_warp), last - first);
  };
  const size_t count_smem = (size_t)kSmWarps * (std::min(K, 32u) + 1) * 128;
  for (uint32_t first = 0; first < n; first += 65535, ++*launched)
    k_class_counts<<<grid_of(first, std::min(n, first + 65535), 1), kSmThreads, count_smem, st>>>(labels, imgs, first, K, c,
                                                                                               err);
  k_class_prefix<<<n, kSmThreads, 0, st>>>(imgs, K, bsz, c, draw0, tot, n_draws, slots, pl.stride);
  PD_CUDA(cudaGetLastError());
  for (uint32_t first = 0; first < n;) {
    uint32_t last = first + 1;  // a group: up to the next image whose draws start over
    while (last < n && last - first < 65535 && h[last].draw_off != 0) last++;
    k_mt_draws<<<last - first, kMtThreads, 0, st>>>(imgs, first, crc, s->seed, n_draws, draws);
    auto res = K < 16 ? k_reservoir<4> : K <= 32 ? k_reservoir<6> : k_reservoir<8>;
    res<<<grid_of(first, last, kSegRun), kSmThreads, 0, st>>>(labels, imgs, first, K, bsz, boff, c, draw0, draws, pl.stride, slots);
    PD_CUDA(cudaGetLastError());
    *launched += 2;
    first = last;
  }
  uint32_t most = 0;
  for (uint32_t i = 0; i < n; i++) most = std::max(most, h[i].n_pix);
  const bool bitmap = most <= kBitmapPixels;
  const size_t smem = bitmap ? ((size_t)most + 127) / 128 * 16 : (size_t)pl.sort_n * 4;
  auto bucket_samples = bitmap ? k_bucket_samples<true> : k_bucket_samples<false>;
  PD_TRY(allow_smem(ctx, bucket_samples, smem));
  bucket_samples<<<n, kSmThreads, smem, st>>>(imgs, bsz, tot, K, slots, pl.stride, pl.sort_n, out, counts);
  PD_CUDA(cudaGetLastError());
  *launched += 1;
  return PD_OK;
}

// Uploads the descriptor block and launches the kernels on a batch that is
// in device memory.  counts/err stay on the device.
int launch_batch(pd_ctx *ctx, const pd_sampler *s, const SamplerPlan &pl, uint32_t n, const uint8_t *data, const uint8_t *labels, uint32_t *out, uint32_t *counts, const DescLayout &lay,
                 uint8_t *dev_desc, void *host_desc, cudaEvent_t *ev) {
  cudaStream_t st = ctx->stream;
  PD_CUDA(h2d(ctx, dev_desc, host_desc, lay.bytes));
  SampImage *imgs = reinterpret_cast<SampImage *>(dev_desc + lay.imgs);
  const uint32_t *item_img = reinterpret_cast<const uint32_t *>(dev_desc + lay.items);
  uint32_t *crc = reinterpret_cast<uint32_t *>(dev_desc + lay.crc);
  uint32_t *cnt = reinterpret_cast<uint32_t *>(dev_desc + lay.count);
  uint32_t *err = reinterpret_cast<uint32_t *>(dev_desc + lay.err);
  int sms = 0, per_sm = 0;
  PD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  PD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sample_scan, kSmThreads, 0));
  PD_CUDA(cudaEventRecord(ev[0], st));
  // the class-weighted sampler does not need the labelled-pixel counts: checksums only
  const uint32_t n_items = s->kind == PD_SAMPLER_UNIFORM ? lay.n_items : lay.n_crc_items;
  const uint32_t grid = std::max(1u, std::min<uint32_t>(n_items, (uint32_t)(sms * std::max(per_sm, 1))));
  k_sample_scan<<<grid, kSmThreads, 0, st>>>(data, labels, imgs, item_img, n_items, lay.n_crc_items,
                                             reinterpret_cast<const uint32_t *>(dev_desc + lay.shifts), crc, cnt,
                                             err + 2);
  PD_CUDA(cudaGetLastError());
  PD_CUDA(cudaEventRecord(ev[1], st));
  uint64_t launched = 2;
  if (s->kind == PD_SAMPLER_UNIFORM) {
    const uint32_t buckets = std::max(pl.sort_n, kSmThreads);
    const size_t smem = ((size_t)s->n_samples * 2 + buckets) * 4;
    PD_TRY(allow_smem(ctx, k_sample_uniform, smem));
    k_sample_uniform<<<n, kSmThreads, smem, st>>>(labels, imgs, crc, cnt, s->n_samples, s->seed, buckets, out, counts,
                                                  err);
  } else {
    PD_TRY(launch_class_weighted(ctx, s, pl, n, static_cast<uint8_t *>(host_desc), lay, labels, imgs, crc,
                                 reinterpret_cast<const uint32_t *>(dev_desc + lay.bucket), out, counts, err, &launched));
  }
  PD_CUDA(cudaGetLastError());
  PD_CUDA(cudaEventRecord(ev[2], st));
  ctx->launches += launched;
  ctx->sample_stats.kernel_launches += 2;  // the two phases
  return PD_OK;
}

struct ImagePlace {
  uint64_t data_lo, data_end, lab_off, out_off;
  uint64_t data_bytes;
  uint32_t n_pix;
};

// Fills the pinned descriptor block for images described by (data_lo, data
// bytes, lab_off, n_pix, out_off); group: of their draws (place_draws).
int fill_desc(HostBuf &hb, const SamplerPlan &pl, const std::vector<ImagePlace> &place, uint64_t group,
              DescLayout *lay_out) {
  const uint32_t n = (uint32_t)place.size();
  uint64_t n_crc = 0, n_lab = 0;
  std::vector<uint32_t> slices(n), chunks(n);
  for (uint32_t i = 0; i < n; i++) {
    slices[i] = (uint32_t)((place[i].data_end - place[i].data_lo + kSliceBytes - 1) / kSliceBytes);
    chunks[i] = ((place[i].n_pix + 15) / 16 + kLabVecsPerItem - 1) / kLabVecsPerItem;
    n_crc += slices[i];
    n_lab += chunks[i];
  }
  PD_CHECK(n_crc + n_lab < (1ull << 31), PD_ERR_UNSUPPORTED, "batch too large");
  DescLayout lay(n, (uint32_t)(n_crc + n_lab), (uint32_t)pl.bucket.size());
  lay.n_crc_items = (uint32_t)n_crc;
  PD_TRY(hb.ensure(lay.bytes));
  uint8_t *h = hb.as<uint8_t>();
  SampImage *im = reinterpret_cast<SampImage *>(h + lay.imgs);
  uint32_t *item_img = reinterpret_cast<uint32_t *>(h + lay.items);
  uint32_t *crc = reinterpret_cast<uint32_t *>(h + lay.crc);
  uint32_t *cnt = reinterpret_cast<uint32_t *>(h + lay.count);
  uint32_t ic = 0, il = (uint32_t)n_crc;
  uint64_t segs = 0;
  for (uint32_t i = 0; i < n; i++) {
    const ImagePlace &p = place[i];
    im[i] = SampImage{p.data_lo, p.data_end, p.lab_off, p.out_off, p.n_pix, (p.n_pix + 15) / 16, slices[i], ic, il,
                      (uint32_t)segs, 0};
    segs += (p.n_pix + kSeg - 1) / kSeg;
    for (uint32_t k = 0; k < slices[i]; k++) item_img[ic++] = i;
    for (uint32_t k = 0; k < chunks[i]; k++) item_img[il++] = i;
    // the initial value 0xFFFFFFFF carried past the image bytes, and the final XOR
    // (images of a batch mostly share their size)
    if (i == 0 || p.data_bytes != place[i - 1].data_bytes)
      crc[i] = gf_mul(0xFFFFFFFFu, gf_x8n(p.data_bytes)) ^ 0xFFFFFFFFu;
    else
      crc[i] = crc[i - 1];
    cnt[i] = 0;
  }
  PD_CHECK(segs < (1ull << 31), PD_ERR_UNSUPPORTED, "batch too large");
  place_draws(im, n, group);
  std::memcpy(h + lay.shifts, shift_constants(), 4ull * kShiftWords);
  reinterpret_cast<uint32_t *>(h + lay.err)[0] = kNoError;  // first image with a label above nClasses
  reinterpret_cast<uint32_t *>(h + lay.err)[1] = kNoError;  // first image whose draws hit the block limit
  reinterpret_cast<uint32_t *>(h + lay.err)[2] = 0;         // next work item of the scan
  if (!pl.bucket.empty()) {
    uint32_t *b = reinterpret_cast<uint32_t *>(h + lay.bucket), *off = b + pl.bucket.size(), o = 0;
    for (size_t k = 0; k < pl.bucket.size(); k++) {
      b[k] = pl.bucket[k];
      off[k] = o;
      o += pl.bucket[k];
    }
  }
  *lay_out = lay;
  return PD_OK;
}

int check_errors(const uint32_t *err, uint32_t first, const pd_sampler *s) {
  PD_CHECK(err[0] == kNoError, PD_ERR_INVALID, "image %u has a label above nClasses %u", first + err[0],
           s->n_classes);
  PD_CHECK(err[1] == kNoError, PD_ERR_CUDA, "image %u: the uniform draws hit their block limit", first + err[1]);
  return PD_OK;
}

double event_ms(cudaEvent_t a, cudaEvent_t b) {
  float ms = 0;
  cudaEventElapsedTime(&ms, a, b);
  return ms;
}

}  // namespace
}  // namespace pd

using namespace pd;

extern "C" int pd_sampler_stride(const pd_sampler *s, uint32_t *stride) {
  PD_CHECK(stride, PD_ERR_INVALID, "null output");
  SamplerPlan pl;
  PD_TRY(plan_sampler(s, &pl));
  *stride = pl.stride;
  return PD_OK;
}

extern "C" int pd_sample_get_stats(pd_ctx *ctx, pd_sample_stats *out) {
  PD_CHECK(ctx && out, PD_ERR_INVALID, "null argument");
  *out = ctx->sample_stats;
  return PD_OK;
}

extern "C" int pd_sample(pd_ctx *ctx, const pd_sampler *s, uint32_t n_images, const void *const *images,
                         const uint8_t *const *labels, const uint32_t *widths, const uint32_t *heights,
                         uint32_t stride, uint32_t *samples, uint32_t *counts) {
  const auto t0 = std::chrono::steady_clock::now();
  PD_CHECK(ctx, PD_ERR_INVALID, "null context");
  SamplerPlan pl;
  PD_TRY(plan_sampler(s, &pl));
  PD_CHECK(stride >= pl.stride, PD_ERR_INVALID, "stride %u below the %u samples per image this sampler needs", stride,
           pl.stride);
  ctx->sample_stats = pd_sample_stats{};
  if (n_images == 0) return PD_OK;
  PD_CHECK(images && labels && widths && heights && samples && counts, PD_ERR_INVALID, "null argument");
  PD_CUDA(cudaSetDevice(ctx->device));
  const uint64_t h2d0 = ctx->bytes_h2d, d2h0 = ctx->bytes_d2h;
  // groups of images whose staged bytes stay below a bound
  struct Group {
    uint32_t first, n;
    uint64_t data_cur, lab_cur;
    std::vector<ImagePlace> place;
  };
  std::vector<Group> groups;
  const uint64_t kGroupBytes = ctx->sample_group;
  for (uint32_t first = 0; first < n_images;) {
    Group g;
    g.first = first;
    g.data_cur = g.lab_cur = 0;
    uint32_t last = first;
    for (; last < n_images; last++) {
      PD_CHECK(images[last] && labels[last], PD_ERR_INVALID, "image %u has a null buffer", last);
      const uint64_t np = (uint64_t)widths[last] * heights[last];
      PD_CHECK(widths[last] >= 1 && heights[last] >= 1 && np < (1ull << 31), PD_ERR_UNSUPPORTED,
               "image %u is %ux%u (1 to 2^31-1 pixels)", last, widths[last], heights[last]);
      const uint64_t db = np * s->pixel_bytes;
      PD_CHECK(db < (1ull << 40), PD_ERR_UNSUPPORTED, "image %u too large", last);
      // zeros before the bytes so that the image ends on a 256-byte block (the
      // checksum reads 256-byte blocks counted from the end)
      const uint64_t pad = (256 - db % 256) % 256;
      const uint64_t dsz = pad + db, lsz = (np + 15) / 16 * 16;
      if (last > first && g.data_cur + dsz + g.lab_cur + lsz > kGroupBytes) break;
      g.place.push_back(
          ImagePlace{g.data_cur, g.data_cur + dsz, g.lab_cur, (uint64_t)(last - first) * stride, db, (uint32_t)np});
      g.data_cur += dsz;
      g.lab_cur += lsz;
    }
    g.n = last - first;
    groups.push_back(std::move(g));
    first = last;
  }
  // Two slots: the host stages group k into one while the device copies, scans
  // and draws group k - 1 from the other; a slot's results come back to its
  // pinned buffer and reach the caller when the slot is reused or at the end.
  PD_CUDA(cudaStreamSynchronize(ctx->stream));  // no earlier call still reads a slot
  for (auto &sl : ctx->samp)
    for (cudaEvent_t &e : sl.ev)
      if (!e) PD_CUDA(cudaEventCreate(&e));
  int busy[2] = {-1, -1};
  DescLayout lays[2];
  auto finish = [&](int si) -> int {
    pd_ctx::SampSlot &sl = ctx->samp[si];
    const Group &g = groups[busy[si]];
    busy[si] = -1;
    PD_CUDA(cudaEventSynchronize(sl.ev[3]));
    const uint32_t *ho = sl.h_out.as<uint32_t>();
    const uint32_t *err = ho + (uint64_t)g.n * stride + g.n;
    PD_TRY(check_errors(err, g.first, s));
    std::memcpy(samples + (uint64_t)g.first * stride, ho, (uint64_t)g.n * stride * 4);
    std::memcpy(counts + g.first, ho + (uint64_t)g.n * stride, (uint64_t)g.n * 4);
    ctx->sample_stats.ms_scan += event_ms(sl.ev[0], sl.ev[1]);
    ctx->sample_stats.ms_draw += event_ms(sl.ev[1], sl.ev[2]);
    for (const ImagePlace &p : g.place) {
      ctx->sample_stats.data_bytes += p.data_bytes;
      ctx->sample_stats.label_bytes += p.n_pix;
    }
    return PD_OK;
  };
  auto fail = [&](int rc) {  // nothing of a failed call stays in flight
    cudaStreamSynchronize(ctx->stream);
    return rc;
  };
  for (size_t k = 0; k < groups.size(); k++) {
    const int si = (int)(k % 2);
    pd_ctx::SampSlot &sl = ctx->samp[si];
    if (busy[si] >= 0) {
      const int rc = finish(si);
      if (rc != PD_OK) return fail(rc);
    }
    const Group &g = groups[k];
    const uint32_t n = g.n, first = g.first;
    // staging: data then labels, each image's zero padding included
    PD_TRY(sl.h_data.ensure(g.data_cur + g.lab_cur + 16));
    uint8_t *hd = sl.h_data.as<uint8_t>(), *hl = hd + g.data_cur;
    const unsigned nt = std::max(1u, std::min({16u, std::thread::hardware_concurrency(), n}));
    auto work = [&](unsigned th) {
      for (uint32_t i = th; i < n; i += nt) {
        const ImagePlace &p = g.place[i];
        const uint64_t pad = p.data_end - p.data_lo - p.data_bytes;
        std::memset(hd + p.data_lo, 0, pad);
        std::memcpy(hd + p.data_lo + pad, images[first + i], p.data_bytes);
        std::memcpy(hl + p.lab_off, labels[first + i], p.n_pix);
        std::memset(hl + p.lab_off + p.n_pix, 0, (p.n_pix + 15) / 16 * 16 - p.n_pix);
      }
    };
    {
      std::vector<std::thread> th;
      for (unsigned q = 1; q < nt; q++) th.emplace_back(work, q);
      work(0);
      for (auto &x : th) x.join();
    }
    DescLayout &lay = lays[si];
    PD_TRY(fill_desc(sl.h_desc, pl, g.place, draw_group(ctx), &lay));
    PD_TRY(sl.d_data.ensure(g.data_cur + g.lab_cur + 16));
    PD_TRY(sl.d_desc.ensure(lay.bytes));
    const uint64_t out_words = (uint64_t)n * stride + n;
    PD_TRY(sl.d_out.ensure(out_words * 4 + 16));
    PD_TRY(sl.h_out.ensure(out_words * 4 + 16));
    uint8_t *dd = sl.d_data.as<uint8_t>(), *dl = dd + g.data_cur;
    int rc = upload_bytes(ctx, dd, hd, g.data_cur + g.lab_cur);
    uint32_t *dout = sl.d_out.as<uint32_t>(), *dcnt = dout + (uint64_t)n * stride;
    if (rc == PD_OK) rc = launch_batch(ctx, s, pl, n, dd, dl, dout, dcnt, lay, sl.d_desc.as<uint8_t>(),
                                       sl.h_desc.ptr, sl.ev);
    if (rc != PD_OK) return fail(rc);
    // samples, counts and the two error words into the slot's pinned buffer
    uint32_t *ho = sl.h_out.as<uint32_t>();
    PD_CUDA(d2h(ctx, ho, dout, out_words * 4));
    PD_CUDA(d2h(ctx, ho + out_words, sl.d_desc.as<uint8_t>() + lay.err, 8));
    PD_CUDA(cudaEventRecord(sl.ev[3], ctx->stream));
    busy[si] = (int)k;
  }
  // the last two groups, in order
  for (size_t k = groups.size() >= 2 ? groups.size() - 2 : 0; k < groups.size(); k++) {
    const int si = (int)(k % 2);
    if (busy[si] == (int)k) {
      const int rc = finish(si);
      if (rc != PD_OK) return fail(rc);
    }
  }
  trim_draws(ctx);
  ctx->sample_stats.images = n_images;
  ctx->sample_stats.h2d_bytes = ctx->bytes_h2d - h2d0;
  ctx->sample_stats.d2h_bytes = ctx->bytes_d2h - d2h0;
  ctx->sample_stats.ms_total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return PD_OK;
}

extern "C" int pd_sample_device(pd_ctx *ctx, const pd_sampler *s, uint32_t n_images, const void *images_device,
                                const uint8_t *labels_device, uint32_t width, uint32_t height, uint32_t stride,
                                uint32_t *samples_device, uint32_t *counts_device) {
  const auto t0 = std::chrono::steady_clock::now();
  PD_CHECK(ctx, PD_ERR_INVALID, "null context");
  SamplerPlan pl;
  PD_TRY(plan_sampler(s, &pl));
  PD_CHECK(stride >= pl.stride, PD_ERR_INVALID, "stride %u below the %u samples per image this sampler needs", stride,
           pl.stride);
  ctx->sample_stats = pd_sample_stats{};
  if (n_images == 0) return PD_OK;
  PD_CHECK(images_device && labels_device && samples_device && counts_device, PD_ERR_INVALID, "null argument");
  const uint64_t np = (uint64_t)width * height, db = np * s->pixel_bytes;
  PD_CHECK(width >= 1 && height >= 1 && np < (1ull << 31), PD_ERR_UNSUPPORTED, "images are %ux%u", width, height);
  PD_CHECK(db % 16 == 0 && np % 16 == 0 && ((uintptr_t)images_device % 16) == 0 &&
               ((uintptr_t)labels_device % 16) == 0,
           PD_ERR_UNSUPPORTED,
           "device images need 16-byte aligned buffers and W*H and W*H*pixel_bytes multiples of 16 (pd_sample "
           "takes any size)");
  PD_CUDA(cudaSetDevice(ctx->device));
  const uint64_t h2d0 = ctx->bytes_h2d, d2h0 = ctx->bytes_d2h;
  std::vector<ImagePlace> place(n_images);
  for (uint32_t i = 0; i < n_images; i++)
    place[i] = ImagePlace{i * db, (i + 1) * db, i * np, (uint64_t)i * stride, db, (uint32_t)np};
  DescLayout lay;
  PD_TRY(fill_desc(ctx->h_sm_desc, pl, place, draw_group(ctx), &lay));
  PD_TRY(ctx->sm_desc.ensure(lay.bytes));
  PD_TRY(launch_batch(ctx, s, pl, n_images, static_cast<const uint8_t *>(images_device), labels_device,
                      samples_device, counts_device, lay, ctx->sm_desc.as<uint8_t>(), ctx->h_sm_desc.ptr, ctx->ev));
  uint32_t err[2];
  PD_CUDA(d2h(ctx, err, ctx->sm_desc.as<uint8_t>() + lay.err, 8));
  PD_CUDA(cudaStreamSynchronize(ctx->stream));
  trim_draws(ctx);
  PD_TRY(check_errors(err, 0, s));
  ctx->sample_stats.images = n_images;
  ctx->sample_stats.data_bytes = db * n_images;
  ctx->sample_stats.label_bytes = np * n_images;
  ctx->sample_stats.ms_scan = event_ms(ctx->ev[0], ctx->ev[1]);
  ctx->sample_stats.ms_draw = event_ms(ctx->ev[1], ctx->ev[2]);
  ctx->sample_stats.h2d_bytes = ctx->bytes_h2d - h2d0;
  ctx->sample_stats.d2h_bytes = ctx->bytes_d2h - d2h0;
  ctx->sample_stats.ms_total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return PD_OK;
}
