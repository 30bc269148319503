// RPN ProposalLayer on the device, batched over images:
//   1. decode      anchor + deltas -> clipped box, score (0 for boxes below the minimum size)
//   2. rank + NMS  a cluster of CTAs per image: takes the best boxes a segment of at most 1024 at a
//                  time, marks in a bit matrix which boxes of the segment suppress which, and which the
//                  boxes kept earlier do, iterates the kept set to its fixed point, stops at
//                  post_nms_topn; writes rois (+ scores) and the count
// The host only needs the per-image counts.
//
// Every float operation that decides which boxes are kept is done with the
// rounding of the CPU code it replaces (mini-caffe src/layers/proposal_layer.cpp:
// TransformBBox :14-53, GenerateProposalsCPU :114-148, SortBBox :88-111,
// NonMaximumSuppressionCPU :150-185, RetrieveRoisCPU :187-203): separate
// multiply and add (no FMA), exp() evaluated in double and the product rounded
// to float once, IEEE division.  Boxes with equal scores are ordered by
// proposal index (the CPU quicksort leaves that order unspecified).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <mutex>

#include "../../../include/mcb200_kernels.h"
#include "detection.cuh"
#include "launch_count.h"
#include "sm100.cuh"

namespace mcb200 {
namespace {

using namespace det;
using sm100::grid_dependency_wait;
using sm100::grid_launch_dependents;

constexpr int kMaxCluster = 8;     // CTAs that work on one image

struct Workspace {
  float4* boxes;                 // [batch][n]     decoded boxes, proposal order
  float* scores;                 // [batch][score_ld]
  uint32_t* score_keys;          // [batch][score_ld]   ascending keys of the descending scores
  float4* kept_boxes;            // [batch][kept], then the areas; used when they do not fit in shared memory
  int n, k;
  int kept;                      // boxes an image can keep: the smaller of post_nms_topn and k
  int score_ld;                  // floats between two images' scores: rows start on 16 bytes
};

size_t align_up(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

// Bytes of one image's kept list: boxes, then areas.
__host__ __device__ inline size_t kept_bytes(int kept) {
  return (static_cast<size_t>(kept) * (sizeof(float4) + sizeof(float)) + 15) & ~static_cast<size_t>(15);
}

size_t carve(const mcb200_proposal_params& p, int batch, char* base, Workspace* ws) {
  const int n = p.num_anchors * p.height * p.width;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* ptr = base ? base + off : nullptr;
    off += align_up(bytes);
    return ptr;
  };
  Workspace w;
  w.n = n;
  w.k = n < p.pre_nms_topn ? n : p.pre_nms_topn;
  w.kept = w.k < p.post_nms_topn ? w.k : p.post_nms_topn;
  w.score_ld = (n + 3) & ~3;
  w.boxes = reinterpret_cast<float4*>(take(sizeof(float4) * n * static_cast<size_t>(batch)));
  w.scores = reinterpret_cast<float*>(take(sizeof(float) * w.score_ld * static_cast<size_t>(batch)));
  w.score_keys = reinterpret_cast<uint32_t*>(take(sizeof(uint32_t) * w.score_ld * static_cast<size_t>(batch)));
  w.kept_boxes = reinterpret_cast<float4*>(take(kept_bytes(w.kept) * batch));
  if (ws) *ws = w;
  return off;
}

// ---------------------------------------------------------------- 1. decode

// A block takes kDecodeCells cells of the map with all their anchors: a warp reads 32 neighbouring
// cells of one anchor (the maps are anchor-major), the results are turned to proposal order (cell-
// major) in shared memory and leave as whole rows.  A group of four boxes'
// values is on its way while the group before it is worked on.
constexpr int kDecodeCells = 64;
constexpr int kDecodeThreads = 256;
constexpr int kDecodeGroup = 4;       // boxes of a thread whose values are asked for together

struct DecodeIn {
  const float* scores;        // foreground scores of image 0; image stride below
  long long score_stride;     // floats between the foreground maps of two images
  const float* deltas;        // [batch][4A][H][W]
  const float* im_info;       // [batch][3]
  const float* anchors;       // [A][4]
};

__global__ void __launch_bounds__(kDecodeThreads, 2)
proposal_decode_kernel(DecodeIn in, mcb200_proposal_params p, Workspace ws, int turned) {
  extern __shared__ __align__(16) unsigned char decode_smem[];
  const int image = blockIdx.y;
  const int hw = p.height * p.width;
  const int n = ws.n;
  const float* score = in.scores + static_cast<size_t>(image) * in.score_stride;
  const float* delta = in.deltas + static_cast<size_t>(image) * 4 * p.num_anchors * hw;
  const float* anchors = in.anchors;
  float4* s_box = reinterpret_cast<float4*>(decode_smem);
  float* s_score = reinterpret_cast<float*>(s_box + (turned ? kDecodeCells * p.num_anchors : 0));
  __shared__ float info[3];
  if (threadIdx.x < 3) info[threadIdx.x] = in.im_info[image * 3 + threadIdx.x];
  const int pos0 = blockIdx.x * kDecodeCells;
  const int items = kDecodeCells * p.num_anchors;
  grid_launch_dependents();
  float in_flight[kDecodeGroup][5];
  auto load = [&](int group) {
#pragma unroll
    for (int u = 0; u < kDecodeGroup; ++u) {
      const int t = group + u * kDecodeThreads;
      const int k = t / kDecodeCells;
      const int pos = pos0 + t % kDecodeCells;
      if (t >= items || pos >= hw) continue;
      in_flight[u][0] = score[k * hw + pos];
#pragma unroll
      for (int j = 0; j < 4; ++j) in_flight[u][1 + j] = delta[(k * 4 + j) * hw + pos];
    }
  };
  load(threadIdx.x);
  __syncthreads();
  const float img_h = info[0], img_w = info[1];
  const float min_size = fmul(static_cast<float>(p.min_size), info[2]);
  for (int group = threadIdx.x; group < items; group += kDecodeGroup * kDecodeThreads) {
#pragma unroll
   for (int u = 0; u < kDecodeGroup; ++u) {
    const int t = group + u * kDecodeThreads;
    if (t >= items) break;
    const float score_here = in_flight[u][0], dx = in_flight[u][1], dy = in_flight[u][2], dlw = in_flight[u][3],
                dlh = in_flight[u][4];
    const int k = t / kDecodeCells;
    const int pos = pos0 + t % kDecodeCells;
    if (pos >= hw) continue;
    const int y = pos / p.width;
    const int x = pos - y * p.width;
    const float fx = static_cast<float>(x * p.feat_stride);
    const float fy = static_cast<float>(y * p.feat_stride);
    float b0 = fadd(fx, anchors[k * 4 + 0]);
    float b1 = fadd(fy, anchors[k * 4 + 1]);
    float b2 = fadd(fx, anchors[k * 4 + 2]);
    float b3 = fadd(fy, anchors[k * 4 + 3]);
    const float w = fadd(fsub(b2, b0), 1.f);
    const float h = fadd(fsub(b3, b1), 1.f);
    const float ctr_x = fadd(b0, fmul(0.5f, w));
    const float ctr_y = fadd(b1, fmul(0.5f, h));
    const float pred_ctr_x = fadd(fmul(dx, w), ctr_x);
    const float pred_ctr_y = fadd(fmul(dy, h), ctr_y);
    // exp in double, product in double, one rounding to float.
    const float pred_w = static_cast<float>(__dmul_rn(exp(static_cast<double>(dlw)), static_cast<double>(w)));
    const float pred_h = static_cast<float>(__dmul_rn(exp(static_cast<double>(dlh)), static_cast<double>(h)));
    b0 = fsub(pred_ctr_x, fmul(0.5f, pred_w));
    b1 = fsub(pred_ctr_y, fmul(0.5f, pred_h));
    b2 = fadd(pred_ctr_x, fmul(0.5f, pred_w));
    b3 = fadd(pred_ctr_y, fmul(0.5f, pred_h));
    const float max_x = fsub(img_w, 1.f);
    const float max_y = fsub(img_h, 1.f);
    b0 = fmaxf(0.f, fminf(b0, max_x));
    b1 = fmaxf(0.f, fminf(b1, max_y));
    b2 = fmaxf(0.f, fminf(b2, max_x));
    b3 = fmaxf(0.f, fminf(b3, max_y));
    const float box_w = fadd(fsub(b2, b0), 1.f);
    const float box_h = fadd(fsub(b3, b1), 1.f);
    const int valid = (box_w >= min_size) && (box_h >= min_size);
    const float s = fmul(static_cast<float>(valid), score_here);

    const float4 box = make_float4(b0, b1, b2, b3);
    const int local = (pos - pos0) * p.num_anchors + k;   // proposal order: (y, x, anchor)
    if (turned) {
      s_box[local] = box;
      s_score[local] = s;
    } else {
      const size_t o = static_cast<size_t>(pos0) * p.num_anchors + local;
      ws.boxes[static_cast<size_t>(image) * n + o] = box;
      ws.scores[static_cast<size_t>(image) * ws.score_ld + o] = s;
      ws.score_keys[static_cast<size_t>(image) * ws.score_ld + o] = descending_key(s);
    }
   }
   load(group + kDecodeGroup * kDecodeThreads);
  }
  if (!turned) return;
  __syncthreads();
  const int here = min(kDecodeCells, hw - pos0) * p.num_anchors;
  float4* box_row = ws.boxes + static_cast<size_t>(image) * n + static_cast<size_t>(pos0) * p.num_anchors;
  const size_t row = static_cast<size_t>(image) * ws.score_ld + static_cast<size_t>(pos0) * p.num_anchors;
  float* score_row = ws.scores + row;
  uint32_t* key_row = ws.score_keys + row;
  for (int t = threadIdx.x; t < here; t += kDecodeThreads) {
    box_row[t] = s_box[t];
    score_row[t] = s_score[t];
    key_row[t] = descending_key(s_score[t]);
  }
}

// ---------------------------------------------------------------- 2a. overlap test

__device__ __forceinline__ float box_area(const float4& b) {
  return fmul(fadd(fsub(b.z, b.x), 1.f), fadd(fsub(b.w, b.y), 1.f));
}

// Decides IoU > threshold ("+1 pixel" convention) as the CPU code does: areas[i] + areas[j] -
// inter, IEEE division.  The division (some forty instructions) runs only where it can matter:
// with `below` = threshold * (1 - 2^-20) and `above` = threshold * (1 + 2^-20), a float product of
// either with the union is off by 2^-24 of itself, so an intersection beyond them decides the
// comparison whatever the quotient's rounding.  A threshold <= 0 or a union that is not a positive
// finite number passes neither test and takes the division.
struct OverlapTest {
  float threshold, below, above;
  __device__ explicit OverlapTest(float thr)
      : threshold(thr), below(thr > 0.f ? fmul(thr, 1.f - 0x1p-20f) : -1.f),
        above(thr > 0.f ? fmul(thr, 1.f + 0x1p-20f) : __builtin_huge_valf()) {}
  // 1: overlaps by more than the threshold; 0: does not; 2: only the division can tell.
  __device__ __forceinline__ int quick(const float4& a, float area_a, const float4& b, float area_b) const {
    const float x1 = fmaxf(a.x, b.x);
    const float y1 = fmaxf(a.y, b.y);
    const float x2 = fminf(a.z, b.z);
    const float y2 = fminf(a.w, b.w);
    const float w = fmaxf(0.f, fadd(fsub(x2, x1), 1.f));
    const float h = fmaxf(0.f, fadd(fsub(y2, y1), 1.f));
    const float inter = fmul(w, h);
    const float uni = fsub(fadd(area_a, area_b), inter);
    return inter < fmul(below, uni) ? 0 : (uni > 0.f && inter > fmul(above, uni)) ? 1 : 2;
  }
  __device__ __noinline__ bool exact(float4 a, float area_a, float4 b, float area_b) const {
    const float w = fmaxf(0.f, fadd(fsub(fminf(a.z, b.z), fmaxf(a.x, b.x)), 1.f));
    const float h = fmaxf(0.f, fadd(fsub(fminf(a.w, b.w), fmaxf(a.y, b.y)), 1.f));
    const float inter = fmul(w, h);
    return fdiv(inter, fsub(fadd(area_a, area_b), inter)) > threshold;
  }
  __device__ __forceinline__ bool operator()(const float4& a, float area_a, const float4& b, float area_b) const {
    const int verdict = quick(a, area_a, b, area_b);
    return verdict == 2 ? exact(a, area_a, b, area_b) : verdict == 1;
  }
};

// ---------------------------------------------------------------- 2b. rank + greedy suppression

namespace cg = cooperative_groups;

constexpr int kRankThreads = 1024;
constexpr int kSegment = 1024;       // boxes taken at a time, at most: one per thread
constexpr int kTopBins = 2048;
// Radix levels of a key (score 32 bits, index 32 bits): 11 + 11 + 10 bits of each half.
__device__ __forceinline__ int level_shift(int level) {
  const int in_half = level % 3 == 0 ? 21 : level % 3 == 1 ? 10 : 0;
  return in_half + (level < 3 ? 32 : 0);
}
__device__ __forceinline__ int level_bins(int level) { return level % 3 == 2 ? 1024 : 2048; }

struct RankShared {
  union {
    struct {
      int top[kTopBins];                   // histogram of the first level
      int bins[kTopBins];                  // histogram of a deeper level
    };
    // [w][c]: bit r: box 32 w + r of the segment suppresses its box c (first CTA)
    uint32_t mask[kSegment / 32][kSegment];
  };
  unsigned long long found[kSegment];      // this CTA's finds
  unsigned long long all[kSegment];        // everybody's, in no order
  uint32_t high[kSegment + 4];             // their upper halves, then ones
  unsigned long long sorted[kSegment];
  float4 boxes[kSegment];
  float area[kSegment];
  uint32_t gone[kSegment / 32];            // boxes of the segment that boxes kept earlier suppress (first CTA)
  uint32_t keep[2][kSegment / 32];         // the walk's set, by the round's parity
  int kept_total;
  int part_fill[kMaxCluster];
  int warp_sum[32];
  int found_bin, found_before, found_total;
  int fill;
};

// Adds one key to a histogram.  Lanes of a warp that all hit one bin (the zero scores of boxes
// below the minimum size, say) are combined into one update.
__device__ __forceinline__ void count_key(int* bins, bool live, int bin) {
  const unsigned lanes = __ballot_sync(0xffffffffu, live);
  if (!live) return;
  const int leader = __ffs(lanes) - 1;
  if (__all_sync(lanes, bin == __shfl_sync(lanes, bin, leader))) {
    if ((threadIdx.x & 31) == leader) atomicAdd(&bins[bin], __popc(lanes));
  } else {
    atomicAdd(&bins[bin], 1);
  }
}

// First bin whose inclusive running count (starting from `before`) exceeds `limit`: its number and
// the count in front of it, or found_bin = -1 and the total when there is none.  Whole block.
__device__ void find_bin(RankShared& sh, const int* bins, int count, int before, int limit) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int a = 2 * t < count ? bins[2 * t] : 0;
  const int b = 2 * t < count ? bins[2 * t + 1] : 0;
  int incl = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) sh.warp_sum[warp] = incl;
  if (t == 0) sh.found_bin = -1;
  __syncthreads();
  int base = lane < warp ? sh.warp_sum[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
  const int excl = before + base + incl - (a + b);
  if (excl <= limit && excl + a + b > limit) {
    const bool second = excl + a <= limit;
    sh.found_bin = 2 * t + (second ? 1 : 0);
    sh.found_before = second ? excl + a : excl;
  }
  if (t == kRankThreads - 1) sh.found_total = excl + a + b;
  __syncthreads();
}

// A threshold T such that between `lo` and `hi` of the n keys are <= T (their number goes to
// *count).  It lies on the coarsest bin boundary that the range allows: for ordinary scores the
// first level's bins decide and no further pass over the keys is needed; ties are cut by index.
template <typename KeyAt>
__device__ unsigned long long find_threshold(RankShared& sh, const KeyAt& key_at, int n, int lo, int hi, int* count) {
  unsigned long long prefix = 0;     // the bits of the levels above, in place
  int before = 0;
  for (int level = 0;; ++level) {
    const int shift = level_shift(level);
    const int nbins = level_bins(level);
    const int* bins = sh.top;
    if (level > 0) {
      const int above = level_shift(level - 1);
      for (int i = threadIdx.x; i < nbins; i += kRankThreads) sh.bins[i] = 0;
      __syncthreads();
      for (int base = 0; base < n; base += kRankThreads) {
        const int i = base + threadIdx.x;
        const unsigned long long key = i < n ? key_at(i) : 0ull;
        count_key(sh.bins, i < n && (key >> above) == (prefix >> above),
                  static_cast<int>(key >> shift) & (nbins - 1));
      }
      __syncthreads();
      bins = sh.bins;
    }
    find_bin(sh, bins, nbins, before, hi);
    const int bin = sh.found_bin, in_front = sh.found_before, total = sh.found_total;
    __syncthreads();                 // the found_* words are rewritten by the next call
    if (bin < 0) {                   // everything down to here fits
      *count = total;
      return level == 0 ? kPadKey : prefix | ((1ull << level_shift(level - 1)) - 1ull);
    }
    const unsigned long long start = prefix | (static_cast<unsigned long long>(bin) << shift);
    if (in_front >= lo) {
      *count = in_front;
      return start - 1ull;           // in_front >= lo >= 1: some key lies below `start`
    }
    prefix = start;
    before = in_front;
  }
}

// A cluster of `kCluster` CTAs per image, which share every part of the work that can be shared
// (`part` = this CTA) and keep one copy each of what the others found, so that all of them take the
// same decisions.  The boxes are needed in score order only as far as the greedy walk gets, which is
// usually a few hundred boxes beyond post_nms_topn: so they are taken a segment of at most
// kSegment at a time.  Where a segment ends does not matter as long as it holds the best of what is
// left:
//   select  a sample of the score keys says below which key about kAim boxes lie; every CTA looks
//           through its share of the keys, the finds are exchanged.  When the sample was wrong by too
//           much (ties, for instance) find_threshold cuts exactly.
//   sort    by counting: a key's place is the number of smaller keys.  Some 700 keys against 700 are
//           60 comparisons per thread of the cluster, where a sorting network or a merge of the same
//           keys is a chain of thirty and more dependent exchanges (5-8 us in one block).
//   mark    which box of the segment suppresses which: 32 x 32 boxes per warp, the results gathered in
//           the first CTA's shared memory; and which boxes the ones kept earlier suppress.
//   walk    the first CTA: keep = not gone and not suppressed by a kept box in front, iterated from
//           "all that are not gone" until nothing changes.  A box's bit is final once those in front
//           of it are, so this ends in the sequential algorithm's set, after as many rounds as the
//           longest chain of suppressions is long.  (A walk in steps of 64 boxes against the kept list
//           makes half the tests, but a step is 4000 cycles of dependent instructions and barriers.)
// The kept set is that of the sequential algorithm (src/layers/proposal_layer.cpp:161-186).
// One block per image that sorted all 6000 boxes and walked them with the division in every test
// took 157 + 62 us.
constexpr int kAim = 700;

template <int kCluster>
__global__ void __launch_bounds__(kRankThreads, 1)
proposal_rank_nms_kernel(Workspace ws, float threshold, int post_nms_topn, int kept_in_smem, int first_image,
                         float* __restrict__ rois, float* __restrict__ roi_scores, int* __restrict__ counts) {
  extern __shared__ __align__(16) unsigned char rank_smem[];
  RankShared& sh = *reinterpret_cast<RankShared*>(rank_smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int part = static_cast<int>(cluster.block_rank());
  const int image = blockIdx.x / kCluster;
  const int n = ws.n, k = ws.k;
  const int t = threadIdx.x, lane = t & 31;
  // The kept list: a copy per CTA in shared memory or, when it is too long for that, one in the workspace.
  float4* kept_box = reinterpret_cast<float4*>(
      kept_in_smem ? rank_smem + ((sizeof(RankShared) + 15) & ~static_cast<size_t>(15))
                   : reinterpret_cast<unsigned char*>(ws.kept_boxes) + image * kept_bytes(ws.kept));
  float* kept_area = reinterpret_cast<float*>(kept_box + ws.kept);
  const float4* boxes = ws.boxes + static_cast<size_t>(image) * n;
  const float* scores = ws.scores + static_cast<size_t>(image) * ws.score_ld;
  const uint32_t* keys = ws.score_keys + static_cast<size_t>(image) * ws.score_ld;
  float* out = rois + static_cast<size_t>(image) * post_nms_topn * 5;
  float* out_scores = roi_scores ? roi_scores + static_cast<size_t>(image) * post_nms_topn : nullptr;
  const OverlapTest suppresses(threshold);
  if (t == 0) sh.fill = 0;
  cluster.sync();   // nobody writes to this CTA's shared memory before it runs
  grid_dependency_wait();
  auto key_at = [&](int i) { return (static_cast<unsigned long long>(keys[i]) << 32) | static_cast<uint32_t>(i); };

  // The sample: a key per thread.
  const int stride = max(n / kRankThreads, 1);
  const bool sampled = t * stride < n;
  const uint32_t sample = sampled ? keys[t * stride] : 0u;

  unsigned long long start = 0ull;   // keys below this have been walked
  int walked = 0, kept_total = 0;

  while (walked < k && kept_total < post_nms_topn) {
    // ---- select
    const int hi = min(walked + kSegment, k);
    uint32_t cut = 0xFFFFFFFFu;                    // n <= hi: everything that is left
    if (n > hi) {
      // The upper 22 bits of the `aim`-th smallest sample, by two histograms.
      const long long wanted = walked + min(kAim, (hi - walked) * 5 / 8);
      const int aim = max(1, static_cast<int>(wanted * min(kRankThreads, n) / n));
      uint32_t prefix = 0u;
      int before = 0;
#pragma unroll
      for (int level = 0; level < 2; ++level) {
        const int shift = level == 0 ? 21 : 10;
        for (int i = t; i < kTopBins; i += kRankThreads) sh.top[i] = 0;
        __syncthreads();
        if (sampled && (level == 0 || (sample >> 21) == (prefix >> 21))) atomicAdd(&sh.top[(sample >> shift) & (kTopBins - 1)], 1);
        __syncthreads();
        find_bin(sh, sh.top, kTopBins, before, aim - 1);
        prefix |= static_cast<uint32_t>(sh.found_bin) << shift;
        before = sh.found_before;
        __syncthreads();
      }
      cut = prefix | 1023u;
    }
    unsigned long long last = (static_cast<unsigned long long>(cut) << 32) | 0xFFFFFFFFull;
    {
      const uint32_t floor_key = static_cast<uint32_t>(start >> 32);
      auto take = [&](uint32_t score_bits, int at) {
        if (score_bits <= cut && score_bits >= floor_key && at < n) {
          const unsigned long long key = (static_cast<unsigned long long>(score_bits) << 32) | static_cast<uint32_t>(at);
          if (key < start) return;
          const int slot = atomicAdd(&sh.fill, 1);
          if (slot < kSegment) sh.found[slot] = key;
        }
      };
      constexpr int kQuads = 3;
      for (int base = 0; base < n; base += kQuads * 4 * kCluster * kRankThreads) {
        uint4 v[kQuads];
#pragma unroll
        for (int u = 0; u < kQuads; ++u) {
          const int i = base + ((u * kCluster + part) * kRankThreads + t) * 4;
          v[u] = i < n ? *reinterpret_cast<const uint4*>(keys + i) : make_uint4(~0u, ~0u, ~0u, ~0u);
        }
#pragma unroll
        for (int u = 0; u < kQuads; ++u) {
          const int i = base + ((u * kCluster + part) * kRankThreads + t) * 4;
          if (min(min(v[u].x, v[u].y), min(v[u].z, v[u].w)) > cut) continue;
          take(v[u].x, i);
          take(v[u].y, i + 1);
          take(v[u].z, i + 2);
          take(v[u].w, i + 3);
        }
      }
    }
    __syncthreads();
    if (t < kCluster) cluster.map_shared_rank(sh.part_fill, t)[part] = sh.fill;
    cluster.sync();
    int m = 0, in_front = 0;
#pragma unroll
    for (int j = 0; j < kCluster; ++j) {
      if (j < part) in_front += sh.part_fill[j];
      m += sh.part_fill[j];
    }
    if (m == 0 || walked + m > hi || (walked > 0 && hi == k && k < n)) {
      // The sample misled, or the cut at pre_nms_topn itself has come: exactly, every CTA by itself.
      for (int i = t; i < kTopBins; i += kRankThreads) sh.top[i] = 0;
      __syncthreads();
      for (int base = 0; base < n; base += kRankThreads) {
        const int i = base + t;
        count_key(sh.top, i < n, i < n ? static_cast<int>(keys[i] >> 21) : 0);
      }
      if (t == 0) sh.fill = 0;
      __syncthreads();
      int count = 0;
      const int lo = k - walked <= kSegment ? k : walked + kSegment / 2;
      last = find_threshold(sh, key_at, n, lo, hi, &count);
      // (the order of the finds differs from CTA to CTA: each ranks all of them)
      for (int i = t; i < n; i += kRankThreads) {
        const unsigned long long key = key_at(i);
        if (key >= start && key <= last) sh.all[atomicAdd(&sh.fill, 1)] = key;
      }
      __syncthreads();
      m = count - walked;
      for (int i = t; i < m; i += kRankThreads) {
        const unsigned long long key = sh.all[i];
        int place = 0;
        for (int q = 0; q < m; ++q) place += sh.all[q] < key ? 1 : 0;
        sh.sorted[place] = key;
      }
    } else {
      // Everybody's finds to everybody.
      for (int i = t; i < sh.part_fill[part]; i += kRankThreads) {
        const unsigned long long key = sh.found[i];
#pragma unroll
        for (int j = 0; j < kCluster; ++j) {
          cluster.map_shared_rank(sh.all, j)[in_front + i] = key;
          cluster.map_shared_rank(sh.high, j)[in_front + i] = static_cast<uint32_t>(key >> 32);
        }
      }
      if (t < 4) sh.high[m + t] = 0xFFFFFFFFu;
      cluster.sync();
      // ---- sort: `helpers` threads count for one key of this CTA's share, four keys at a time by
      // their upper halves (equal ones, a rare sight, are told apart in a second pass)
      const int share = (m + kCluster - 1) / kCluster;
      int helpers = 32;
      while (helpers > 1 && share * helpers > kRankThreads) helpers >>= 1;
      const int sub = t & (helpers - 1);
      for (int base = 0; base < share; base += kRankThreads / helpers) {
        const int local = base + t / helpers;
        const int at = part * share + local;
        const bool mine = local < share && at < m;
        const unsigned long long key = mine ? sh.all[at] : 0ull;
        const uint32_t h = static_cast<uint32_t>(key >> 32);
        int below = 0, upto = 0;
#pragma unroll 4
        for (int q = sub * 4; q < m; q += helpers * 4) {
          const uint4 v = *reinterpret_cast<const uint4*>(sh.high + q);
          below += (v.x < h ? 1 : 0) + (v.y < h ? 1 : 0) + (v.z < h ? 1 : 0) + (v.w < h ? 1 : 0);
          upto += (v.x <= h ? 1 : 0) + (v.y <= h ? 1 : 0) + (v.z <= h ? 1 : 0) + (v.w <= h ? 1 : 0);
        }
        for (int o = helpers >> 1; o > 0; o >>= 1) {
          below += __shfl_xor_sync(0xffffffffu, below, o);
          upto += __shfl_xor_sync(0xffffffffu, upto, o);
        }
        if (mine && upto != below + 1) {
          below = 0;
          for (int q = 0; q < m; ++q) below += sh.all[q] < key ? 1 : 0;
        }
        for (int j = sub; j < kCluster; j += helpers) {
          if (mine) cluster.map_shared_rank(sh.sorted, j)[below] = key;
        }
      }
    }
    cluster.sync();
    if (t < m) {
      const float4 b = boxes[sh.sorted[t] & 0xFFFFFFFFull];
      sh.boxes[t] = b;
      sh.area[t] = box_area(b);
    }
    if (t < kSegment / 32) sh.gone[t] = 0u;
    if (t == 0) sh.fill = 0;
    cluster.sync();

    // ---- mark
    const int blocks = (m + 31) >> 5;
    const int crew = kCluster * (kRankThreads / 32);
    uint32_t* mask = cluster.map_shared_rank(&sh.mask[0][0], 0);
    int column_block = 0, first_tile = 0;      // tiles run over column blocks, then the row blocks up to it
    for (int tile = (t >> 5) * kCluster + part; tile < blocks * (blocks + 1) / 2; tile += crew) {
      while (tile > first_tile + column_block) first_tile += ++column_block;
      const int w = tile - first_tile;
      const int c = column_block * 32 + lane;
      const float4 b = sh.boxes[c];
      const float area_b = sh.area[c];
      const int rows = min(32, m - w * 32);
      uint32_t bits = 0u, unsure = 0u;
#pragma unroll 4
      for (int r = 0; r < rows; ++r) {
        const int verdict = suppresses.quick(sh.boxes[w * 32 + r], sh.area[w * 32 + r], b, area_b);
        bits |= static_cast<uint32_t>(verdict & 1) << r;
        unsure |= static_cast<uint32_t>(verdict >> 1) << r;
      }
      for (; unsure; unsure &= unsure - 1) {
        const int r = __ffs(unsure) - 1;
        if (suppresses.exact(sh.boxes[w * 32 + r], sh.area[w * 32 + r], b, area_b)) bits |= 1u << r;
      }
      if (w == column_block) bits &= (1u << lane) - 1u;   // only boxes in front suppress
      if (c < m) mask[w * kSegment + c] = bits;
    }
    if (kept_total > 0) {
      uint32_t* gone = cluster.map_shared_rank(sh.gone, 0);
      for (int task = (t >> 5) * kCluster + part; task < blocks * 8; task += crew) {
        const int c = (task >> 3) * 32 + lane;
        const float4 b = sh.boxes[c];
        const float area_b = sh.area[c];
        bool hit = false;
        for (int q = task & 7; q < kept_total; q += 8) hit = hit || suppresses(kept_box[q], kept_area[q], b, area_b);
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (lane == 0 && hits) atomicOr(gone + (task >> 3), hits);
      }
    }
    cluster.sync();

    // ---- walk
    if (part == 0) {
      const int own = t >> 5;
      uint32_t busy = 0u;                     // words of this column that suppress anything at all
      if (t < m) {
        for (int w = 0; w <= own; ++w) busy |= (sh.mask[w][t] != 0u ? 1u : 0u) << w;
      }
      const bool alive = t < m && !((sh.gone[own] >> lane) & 1u);
      uint32_t word = __ballot_sync(0xffffffffu, alive);
      if (lane == 0) sh.keep[0][own] = word;
      __syncthreads();
      for (int round = 0;; round ^= 1) {
        bool stays = alive;
        for (uint32_t left = busy; left && stays; left &= left - 1) {
          const int w = __ffs(left) - 1;
          stays = !(sh.mask[w][t] & sh.keep[round][w]);
        }
        const uint32_t next = __ballot_sync(0xffffffffu, stays);
        if (lane == 0) sh.keep[round ^ 1][own] = next;
        const int changed = __syncthreads_or(next != word);
        word = next;
        if (!changed) break;
      }
      // (both copies of the set are the same now)
      int before = kept_total;
      for (int w = 0; w < own; ++w) before += __popc(sh.keep[0][w]);
      const int pos = before + __popc(word & ((1u << lane) - 1u));
      const bool more = walked + m < k;       // the others need the kept boxes for the next segment
      if (((word >> lane) & 1u) && pos < post_nms_topn) {
        const float4 kept = sh.boxes[t];
#pragma unroll
        for (int j = 0; j < kCluster; ++j) {
          if (kept_in_smem && more) {
            cluster.map_shared_rank(kept_box, j)[pos] = kept;
            cluster.map_shared_rank(kept_area, j)[pos] = sh.area[t];
          }
        }
        if (!kept_in_smem) {
          kept_box[pos] = kept;
          kept_area[pos] = sh.area[t];
        }
        out[pos * 5 + 0] = static_cast<float>(first_image + image);
        out[pos * 5 + 1] = kept.x;
        out[pos * 5 + 2] = kept.y;
        out[pos * 5 + 3] = kept.z;
        out[pos * 5 + 4] = kept.w;
        if (out_scores) out_scores[pos] = scores[sh.sorted[t] & 0xFFFFFFFFull];
      }
      if (t == kRankThreads - 1) {
        const int total = min(before + __popc(word), post_nms_topn);
#pragma unroll
        for (int j = 0; j < kCluster; ++j) *cluster.map_shared_rank(&sh.kept_total, j) = total;
      }
    }
    cluster.sync();
    kept_total = sh.kept_total;
    walked += m;
    start = last + 1ull;
  }
  if (t == 0 && part == 0) counts[image] = kept_total;
}

}  // namespace
}  // namespace mcb200

using namespace mcb200;

static int validate(const mcb200_proposal_params* p, int batch) {
  if (!p || batch < 1) return -1;
  if (p->num_anchors < 1 || p->height < 1 || p->width < 1 || p->feat_stride < 1 || p->pre_nms_topn < 1 ||
      p->post_nms_topn < 1)
    return -2;
  const long long n = static_cast<long long>(p->num_anchors) * p->height * p->width;
  if (n > (1 << 24)) return -3;
  const int k = n < p->pre_nms_topn ? static_cast<int>(n) : p->pre_nms_topn;
  if (det::next_pow2(k) > 16384) return -4;
  return 0;
}

// Dynamic shared memory a block may ask for.
constexpr size_t kRankSharedLimit = 220 * 1024;
constexpr size_t kDecodeSharedLimit = 48 * 1024;

// The ranking kernel uses more dynamic shared memory than a kernel gets by default; the opt-in is per device and is made on a device's first call
// (nets on several host threads may make that call at the same time).
static cudaError_t configure_kernels() {
  static bool configured[64] = {false};
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (dev < 0 || dev >= 64 || configured[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(proposal_rank_nms_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kRankSharedLimit));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(proposal_rank_nms_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kRankSharedLimit));
  if (e != cudaSuccess) return e;
  configured[dev] = true;
  return cudaSuccess;
}

// Moves the valid rows of images 1 .. batch-1 up against those of the image in
// front (rows of image b start at b * post and move to the sum of the counts
// before it).  A row never moves to a higher address and images are handled in
// order, so what is overwritten has been moved already; inside an image the
// block copies `blockDim.x` values at a time, reading a piece completely before
// writing it (source and destination ranges may overlap).
static __global__ void proposal_compact_kernel(float* __restrict__ rois, float* __restrict__ roi_scores,
                                        const int* __restrict__ counts, int batch, int post) {
  int total = counts[0];
  for (int b = 1; b < batch; ++b) {
    const int rows = counts[b];
    if (rows > 0 && total != b * post) {
      for (int pass = 0; pass < 2; ++pass) {
        float* base = pass == 0 ? rois : roi_scores;
        if (!base) continue;
        const int width = pass == 0 ? 5 : 1;
        const float* src = base + static_cast<size_t>(b) * post * width;
        float* dst = base + static_cast<size_t>(total) * width;
        const int values = rows * width;
        for (int i0 = 0; i0 < values; i0 += blockDim.x) {
          const int i = i0 + threadIdx.x;
          const float v = i < values ? src[i] : 0.f;
          __syncthreads();
          if (i < values) dst[i] = v;
          __syncthreads();
        }
      }
    }
    total += rows;
  }
}

extern "C" size_t mcb200_proposal_workspace_bytes(const mcb200_proposal_params* p, int batch) {
  if (validate(p, batch) != 0) return 0;
  return carve(*p, batch, nullptr, nullptr);
}

extern "C" int mcb200_proposal_forward_from(const mcb200_proposal_params* p, int first_image, int batch,
                                            const float* fg_scores, long long score_stride, const float* deltas, const float* im_info,
                                            const float* anchors, void* workspace, float* rois, float* roi_scores,
                                            int* counts, void* stream) {
  const int rc = validate(p, batch);
  if (rc != 0) return rc;
  if (!fg_scores || !deltas || !im_info || !anchors || !workspace || !rois || !counts) return -5;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return -6;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const cudaError_t configured = configure_kernels();
  if (configured != cudaSuccess) return static_cast<int>(configured);
  Workspace ws;
  carve(*p, batch, static_cast<char*>(workspace), &ws);

  {
    const int hw = p->height * p->width;
    const size_t smem = static_cast<size_t>(kDecodeCells) * p->num_anchors * (sizeof(float4) + sizeof(float));
    const int turned = smem <= kDecodeSharedLimit ? 1 : 0;
    const DecodeIn in = {fg_scores, score_stride, deltas, im_info, anchors};
    proposal_decode_kernel<<<dim3((hw + kDecodeCells - 1) / kDecodeCells, batch), kDecodeThreads, turned ? smem : 0, st>>>(
        in, *p, ws, turned);
    count_launch();
  }
  // The kept list goes to shared memory where it fits beside the fixed part.
  size_t smem = (sizeof(RankShared) + 15) & ~static_cast<size_t>(15);
  const int kept_in_smem = smem + kept_bytes(ws.kept) <= kRankSharedLimit ? 1 : 0;
  if (kept_in_smem) smem += kept_bytes(ws.kept);
  // Eight CTAs per image while all of them find an SM of their own, else four.
  const int parts = batch * 8 <= 148 ? 8 : 4;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(batch * parts);
  cfg.blockDim = dim3(kRankThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // set-up beside the decode kernel's tail
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = parts;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, parts == 8 ? proposal_rank_nms_kernel<8> : proposal_rank_nms_kernel<4>, ws,
                                           p->nms_thresh, p->post_nms_topn, kept_in_smem, first_image, rois, roi_scores,
                                           counts);
  count_launch();
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

extern "C" int mcb200_proposal_forward(const mcb200_proposal_params* p, int batch, const float* scores,
                                       const float* deltas, const float* im_info, const float* anchors,
                                       void* workspace, float* rois, float* roi_scores, int* counts, void* stream) {
  const int rc = validate(p, batch);
  if (rc != 0) return rc;
  // Foreground scores are the second half of the 2A score channels.
  const long long n = static_cast<long long>(p->num_anchors) * p->height * p->width;
  return mcb200_proposal_forward_from(p, 0, batch, scores ? scores + n : nullptr, 2 * n, deltas, im_info, anchors, workspace,
                                      rois, roi_scores, counts, stream);
}

// The images' row blocks (image b's rows start at b * post) one behind the other in another buffer,
// which may be pinned host memory: one block per image.
static __global__ void __launch_bounds__(256)
proposal_gather_kernel(const float* __restrict__ rois, const float* __restrict__ roi_scores, const int* __restrict__ counts,
                       int post, float* __restrict__ rois_out, float* __restrict__ scores_out) {
  __shared__ int before;
  const int image = blockIdx.x;
  if (threadIdx.x == 0) before = 0;
  __syncthreads();
  int sum = 0;
  for (int i = threadIdx.x; i < image; i += blockDim.x) sum += counts[i];
  if (sum) atomicAdd(&before, sum);
  __syncthreads();
  const int rows = counts[image], first = before;
  const float* src = rois + static_cast<size_t>(image) * post * 5;
  for (int i = threadIdx.x; i < rows * 5; i += blockDim.x) rois_out[static_cast<size_t>(first) * 5 + i] = src[i];
  if (!scores_out) return;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) scores_out[first + i] = roi_scores[static_cast<size_t>(image) * post + i];
}

extern "C" int mcb200_proposal_gather(const float* rois, const float* roi_scores, const int* counts, int batch, int post_nms_topn,
                                      float* rois_out, float* scores_out, void* stream) {
  if (!rois || !counts || !rois_out || (scores_out && !roi_scores) || batch < 1 || post_nms_topn < 1) return -1;
  proposal_gather_kernel<<<batch, 256, 0, static_cast<cudaStream_t>(stream)>>>(rois, roi_scores, counts, post_nms_topn,
                                                                              rois_out, scores_out);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_proposal_compact(float* rois, float* roi_scores, const int* counts, int batch,
                                       int post_nms_topn, void* stream) {
  if (!rois || !counts || batch < 1 || post_nms_topn < 1) return -1;
  if (batch == 1) return 0;
  proposal_compact_kernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(rois, roi_scores, counts, batch,
                                                                             post_nms_topn);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------------ variant without allocation

// Scratch of mcb200_proposal_forward_static.  It lives in the library's device
// image: every GPU that loads the library carries these 8 MiB until the process
// exits.  An image of 65536 proposals takes 1.3 MB of it, one of the stock R-FCN setting (63 x 38
// map, 15 anchors) 0.72 MB; a call whose batch needs more than the array holds
// is refused.
static constexpr size_t kStaticScratchBytes = static_cast<size_t>(8) << 20;
static __device__ __align__(256) unsigned char g_proposal_static_scratch[kStaticScratchBytes];

namespace {

// Device address of the scratch array on the current device, looked up once per device.
// In host code the array's name is only a handle; the address has to be asked for
// with that device current.
int static_scratch(void** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= 64) return -21;
  static void* scratch_of_device[64] = {nullptr};
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (!scratch_of_device[dev]) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_proposal_static_scratch);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (!ptr) return -22;
    scratch_of_device[dev] = ptr;
  }
  *out = scratch_of_device[dev];
  return 0;
}

}  // namespace

extern "C" int mcb200_proposal_static_warmup(void) {
  void* scratch = nullptr;
  const int rc = static_scratch(&scratch);
  if (rc != 0) return rc;
  return static_cast<int>(configure_kernels());
}

extern "C" int mcb200_proposal_forward_static(const mcb200_proposal_params* p, int batch, const float* scores,
                                              const float* deltas, const float* im_info, const float* anchors,
                                              float* rois, float* roi_scores, int* counts, void* stream) {
  const int rc = validate(p, batch);
  if (rc != 0) return rc;
  const size_t need = carve(*p, batch, nullptr, nullptr);
  if (need > kStaticScratchBytes) {
    fprintf(stderr,
            "mcb200_proposal_forward_static: this request needs %zu bytes of scratch, the built-in buffer holds %zu; "
            "use mcb200_proposal_forward with a caller-provided workspace\n",
            need, kStaticScratchBytes);
    return -20;
  }
  void* scratch = nullptr;
  const int found = static_scratch(&scratch);
  if (found != 0) return found;
  // Every scratch word the kernels read is written earlier in the same call
  // (boxes and scores for all proposals, the kept boxes), so nothing has to be cleared between calls.
  return mcb200_proposal_forward(p, batch, scores, deltas, im_info, anchors, scratch, rois, roi_scores, counts,
                                 stream);
}
