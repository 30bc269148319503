// SSD DetectionOutput on the device:
//   A. per (image, class) block: collect priors whose class score passes the
//      confidence threshold, take the top_k best (histogram + bitonic sort in
//      shared memory, ties by prior index like std::stable_sort), decode their
//      boxes, greedy NMS (overlap bit matrix, then the kept set iterated, by the whole block)
//   B. per image block: if more than keep_top_k detections survive, keep the
//      keep_top_k best over all classes; lay the rows out label-ascending
//   C. per image block: prefix sum of the per-image counts, compact the rows
// The host reads back one int (the row count).
//
// Arithmetic follows mini-caffe's CPU code operation by operation so that the
// kept sets agree bit for bit: DecodeBBox (src/util/bbox_util.cpp:242-330;
// centre/size decode with exp() in double, results rounded to float once),
// BBoxSize (:80-98), JaccardOverlap (:184-205), GetMaxScoreIndex (:524-541),
// ApplyNMSFast (:681-716), the keep_top_k step and row layout of
// DetectionOutputLayer::Forward_cpu (src/layers/detection_output_layer.cpp:107-225).
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <mutex>

#include "../../../include/mcb200_kernels.h"
#include "detection.cuh"
#include "launch_count.h"

namespace mcb200 {
namespace {

using namespace det;

struct Entry {       // one kept detection of one (image, class)
  float score;
  float xmin, ymin, xmax, ymax;
};

struct Workspace {
  Entry* entries;    // [batch][classes][per_class]
  int* class_count;  // [batch][classes]
  float* rows;       // [batch][max_rows][7]
  int* image_count;  // [batch]
  int per_class, max_rows;
};

size_t align_up(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

int per_class_limit(const mcb200_detout_params& p) {
  int k = p.top_k < 0 ? p.num_priors : p.top_k;
  if (k > p.num_priors) k = p.num_priors;
  return k;
}

int max_rows(const mcb200_detout_params& p) {
  const int classes = p.num_classes - (p.background_label_id >= 0 && p.background_label_id < p.num_classes ? 1 : 0);
  long long all = static_cast<long long>(classes) * per_class_limit(p);
  if (p.keep_top_k > -1 && p.keep_top_k < all) all = p.keep_top_k;
  return static_cast<int>(all);
}

size_t carve(const mcb200_detout_params& p, int batch, char* base, Workspace* ws) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* ptr = base ? base + off : nullptr;
    off += align_up(bytes);
    return ptr;
  };
  Workspace w;
  w.per_class = per_class_limit(p);
  w.max_rows = max_rows(p);
  w.entries = reinterpret_cast<Entry*>(take(sizeof(Entry) * static_cast<size_t>(batch) * p.num_classes * w.per_class));
  w.class_count = reinterpret_cast<int*>(take(sizeof(int) * static_cast<size_t>(batch) * p.num_classes));
  w.rows = reinterpret_cast<float*>(take(sizeof(float) * 7 * static_cast<size_t>(batch) * (w.max_rows > 0 ? w.max_rows : 1)));
  w.image_count = reinterpret_cast<int*>(take(sizeof(int) * static_cast<size_t>(batch)));
  if (ws) *ws = w;
  return off;
}

// ---------------------------------------------------------------- box arithmetic

struct Box {
  float xmin, ymin, xmax, ymax, size;
};

__device__ __forceinline__ float box_size(float xmin, float ymin, float xmax, float ymax) {
  if (xmax < xmin || ymax < ymin) return 0.f;
  return fmul(fsub(xmax, xmin), fsub(ymax, ymin));
}

__device__ Box decode_box(const mcb200_detout_params& p, const float* prior, const float* var, const float* loc) {
  const float pxmin = prior[0], pymin = prior[1], pxmax = prior[2], pymax = prior[3];
  const float bx0 = loc[0], bx1 = loc[1], bx2 = loc[2], bx3 = loc[3];
  Box b;
  if (p.code_type == 1) {  // CORNER
    if (p.variance_encoded_in_target) {
      b.xmin = fadd(pxmin, bx0);
      b.ymin = fadd(pymin, bx1);
      b.xmax = fadd(pxmax, bx2);
      b.ymax = fadd(pymax, bx3);
    } else {
      b.xmin = fadd(pxmin, fmul(var[0], bx0));
      b.ymin = fadd(pymin, fmul(var[1], bx1));
      b.xmax = fadd(pxmax, fmul(var[2], bx2));
      b.ymax = fadd(pymax, fmul(var[3], bx3));
    }
  } else if (p.code_type == 2) {  // CENTER_SIZE
    const float pw = fsub(pxmax, pxmin);
    const float ph = fsub(pymax, pymin);
    // (a + b) / 2. is evaluated in double and rounded to float.
    const float pcx = static_cast<float>(__ddiv_rn(static_cast<double>(fadd(pxmin, pxmax)), 2.0));
    const float pcy = static_cast<float>(__ddiv_rn(static_cast<double>(fadd(pymin, pymax)), 2.0));
    float cx, cy, w, h;
    if (p.variance_encoded_in_target) {
      cx = fadd(fmul(bx0, pw), pcx);
      cy = fadd(fmul(bx1, ph), pcy);
      w = static_cast<float>(__dmul_rn(exp(static_cast<double>(bx2)), static_cast<double>(pw)));
      h = static_cast<float>(__dmul_rn(exp(static_cast<double>(bx3)), static_cast<double>(ph)));
    } else {
      cx = fadd(fmul(fmul(var[0], bx0), pw), pcx);
      cy = fadd(fmul(fmul(var[1], bx1), ph), pcy);
      w = static_cast<float>(__dmul_rn(exp(static_cast<double>(fmul(var[2], bx2))), static_cast<double>(pw)));
      h = static_cast<float>(__dmul_rn(exp(static_cast<double>(fmul(var[3], bx3))), static_cast<double>(ph)));
    }
    // centre -+ size / 2. : double subtraction, one rounding to float.
    const double hw = __ddiv_rn(static_cast<double>(w), 2.0);
    const double hh = __ddiv_rn(static_cast<double>(h), 2.0);
    b.xmin = static_cast<float>(__dsub_rn(static_cast<double>(cx), hw));
    b.ymin = static_cast<float>(__dsub_rn(static_cast<double>(cy), hh));
    b.xmax = static_cast<float>(__dadd_rn(static_cast<double>(cx), hw));
    b.ymax = static_cast<float>(__dadd_rn(static_cast<double>(cy), hh));
  } else {  // CORNER_SIZE
    const float pw = fsub(pxmax, pxmin);
    const float ph = fsub(pymax, pymin);
    if (p.variance_encoded_in_target) {
      b.xmin = fadd(pxmin, fmul(bx0, pw));
      b.ymin = fadd(pymin, fmul(bx1, ph));
      b.xmax = fadd(pxmax, fmul(bx2, pw));
      b.ymax = fadd(pymax, fmul(bx3, ph));
    } else {
      b.xmin = fadd(pxmin, fmul(fmul(var[0], bx0), pw));
      b.ymin = fadd(pymin, fmul(fmul(var[1], bx1), ph));
      b.xmax = fadd(pxmax, fmul(fmul(var[2], bx2), pw));
      b.ymax = fadd(pymax, fmul(fmul(var[3], bx3), ph));
    }
  }
  b.size = box_size(b.xmin, b.ymin, b.xmax, b.ymax);
  return b;
}

// Jaccard overlap of normalised boxes; 0 when they do not intersect.
__device__ __forceinline__ float jaccard(const Box& a, const Box& b) {
  if (b.xmin > a.xmax || b.xmax < a.xmin || b.ymin > a.ymax || b.ymax < a.ymin) return 0.f;
  const float ixmin = fmaxf(a.xmin, b.xmin);
  const float iymin = fmaxf(a.ymin, b.ymin);
  const float ixmax = fminf(a.xmax, b.xmax);
  const float iymax = fminf(a.ymax, b.ymax);
  const float iw = fsub(ixmax, ixmin);
  const float ih = fsub(iymax, iymin);
  if (iw > 0.f && ih > 0.f) {
    const float isize = fmul(iw, ih);
    return fdiv(isize, fsub(fadd(a.size, b.size), isize));
  }
  return 0.f;
}

// ---------------------------------------------------------------- the k best of many keys

constexpr int kBins = 2048;
constexpr int kEdge = 1024;

// Shared memory of one selection.
struct SelectShared {
  int bins[kBins];
  unsigned long long edge[kEdge];   // the keys of the bin that holds the k-th
  int warp_sum[32];
  uint32_t low, high;               // range of the keys' upper halves
  int bin, before, edges;
  unsigned long long threshold;
  int hist[256];                    // the radix walk's
  unsigned long long bcast[2];
};

// A threshold T such that exactly k of the keys are <= T (k smaller than their number).  The upper
// halves, which `each` hands to its callback one by one, are spread over kBins equal steps of their own
// range [low, high] (scores of one layer share sign and most exponent bits: bins cut from the top bits
// would hold thousands each); the keys of the bin that the k-th falls into are ranked by counting.
// Only when that bin holds more than kEdge (ties) the radix walk over `fetch(0 .. n - 1)` decides.
// Whole block; sh.low / sh.high are set by the caller.
template <typename Each, typename Fetch>
__device__ unsigned long long select_threshold(SelectShared& sh, const Each& each, const Fetch& fetch, int n, int k) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, threads = blockDim.x;
  const uint32_t low = sh.low, range = sh.high - sh.low;
  const int shift = max(0, 32 - __clz(range) - 11);       // range >> shift < kBins
  for (int i = t; i < kBins; i += threads) sh.bins[i] = 0;
  if (t == 0) sh.edges = 0;
  __syncthreads();
  each([&](unsigned long long key) { atomicAdd(&sh.bins[(static_cast<uint32_t>(key >> 32) - low) >> shift], 1); });
  __syncthreads();
  // First bin whose running count reaches k.
  const int per = kBins / threads;
  int own = 0;
  for (int j = 0; j < per; ++j) own += sh.bins[t * per + j];
  int incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) sh.warp_sum[warp] = incl;
  __syncthreads();
  int base = lane < warp ? sh.warp_sum[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
  int before = base + incl - own;
  if (before < k && before + own >= k) {
    int bin = t * per;
    while (before + sh.bins[bin] < k) before += sh.bins[bin++];
    sh.bin = bin;
    sh.before = before;
  }
  __syncthreads();
  const uint32_t bin = sh.bin;
  const int wanted = k - sh.before;
  if (sh.bins[bin] > kEdge) return block_kth_smallest(fetch, n, k, sh.hist, sh.bcast);
  each([&](unsigned long long key) {
    if (((static_cast<uint32_t>(key >> 32) - low) >> shift) == bin) sh.edge[atomicAdd(&sh.edges, 1)] = key;
  });
  __syncthreads();
  const int edges = sh.edges;
  for (int i = t; i < edges; i += threads) {
    const unsigned long long key = sh.edge[i];
    int rank = 1;
    for (int q = 0; q < edges; ++q) rank += sh.edge[q] < key ? 1 : 0;
    if (rank == wanted) sh.threshold = key;
  }
  __syncthreads();
  return sh.threshold;
}

// Range of the upper halves over the block, into sh.low / sh.high (a barrier follows before use).
__device__ __forceinline__ void note_range(SelectShared& sh, uint32_t low, uint32_t high) {
  low = __reduce_min_sync(0xffffffffu, low);
  high = __reduce_max_sync(0xffffffffu, high);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&sh.low, low);
    atomicMax(&sh.high, high);
  }
}

// ---------------------------------------------------------------- A. per (image, class)

constexpr int kClassThreads = 512;
constexpr uint32_t kNoKey = 0xFFFFFFFFu;   // the key of no score that passes a comparison (a NaN's)

// Overlap > threshold without the division where a product decides (a float product of the threshold
// widened by 2^-20 either way is off by 2^-24 of itself; in between, and for thresholds <= 0, the
// quotient is compared).
struct JaccardTest {
  float threshold, below, above;
  __device__ explicit JaccardTest(float thr)
      : threshold(thr), below(thr > 0.f ? fmul(thr, 1.f - 0x1p-20f) : -1.f),
        above(thr > 0.f ? fmul(thr, 1.f + 0x1p-20f) : __builtin_huge_valf()) {}
  // 1: more than the threshold; 0: not; 2: only the quotient can tell.  Boxes that do not meet have an
  // intersection of 0 here and pass no threshold >= 0, as in the CPU code.
  __device__ __forceinline__ int quick(const float4& a, float size_a, const float4& b, float size_b) const {
    const float iw = fmaxf(fsub(fminf(a.z, b.z), fmaxf(a.x, b.x)), 0.f);
    const float ih = fmaxf(fsub(fminf(a.w, b.w), fmaxf(a.y, b.y)), 0.f);
    const float isize = fmul(iw, ih);
    const float uni = fsub(fadd(size_a, size_b), isize);
    return isize < fmul(below, uni) ? 0 : (uni > 0.f && isize > fmul(above, uni)) ? 1 : 2;
  }
};

// Shared memory: the selection's, selected keys [padded], boxes and sizes [padded], kept list [padded], then one
// region for the priors' score keys (4 bytes each, kNoKey where the score does not pass) and, once the
// selection is over, the overlap bits.
struct ClassShared {
  SelectShared select;
  uint32_t keep[2][128];     // the walk's set, by the round's parity
  int num_cand, num_sel;
};

__host__ __device__ inline size_t class_region_bytes(int num_priors, int limit) {
  const size_t keys = static_cast<size_t>(num_priors) * sizeof(uint32_t);
  const size_t bits = limit <= 1024 ? static_cast<size_t>((limit + 31) / 32) * limit * sizeof(uint32_t) : 0;
  return keys > bits ? keys : bits;
}

__global__ void __launch_bounds__(kClassThreads, 2)
detout_class_kernel(const float* __restrict__ loc, const float* __restrict__ conf, const float* __restrict__ prior,
                    mcb200_detout_params p, Workspace ws, int padded, float eta) {
  extern __shared__ __align__(16) unsigned char class_smem[];
  ClassShared& sh = *reinterpret_cast<ClassShared*>(class_smem);
  unsigned long long* sel = reinterpret_cast<unsigned long long*>(class_smem + ((sizeof(ClassShared) + 15) & ~static_cast<size_t>(15)));
  float4* corners = reinterpret_cast<float4*>(sel + padded);
  float* sizes = reinterpret_cast<float*>(corners + padded);
  int* kept = reinterpret_cast<int*>(sizes + padded);
  auto box_at = [&](int i) {
    const float4 c = corners[i];
    return Box{c.x, c.y, c.z, c.w, sizes[i]};
  };
  uint32_t* region = reinterpret_cast<uint32_t*>(kept + padded);

  const int cls = blockIdx.x;
  const int image = blockIdx.y;
  const int limit = ws.per_class;
  const int t = threadIdx.x, lane = t & 31;
  int* out_count = ws.class_count + static_cast<size_t>(image) * p.num_classes + cls;
  if (cls == p.background_label_id || limit == 0) {   // top_k 0 keeps nothing: there is no key to cut at
    if (t == 0) *out_count = 0;
    return;
  }
  if (t == 0) {
    sh.num_cand = 0;
    sh.num_sel = 0;
    sh.select.low = 0xFFFFFFFFu;
    sh.select.high = 0u;
  }
  for (int i = t; i < padded; i += kClassThreads) sel[i] = kPadKey;
  __syncthreads();
  const float* scores = conf + static_cast<size_t>(image) * p.num_priors * p.num_classes + cls;
  {
    // The class's column of the score matrix: eight strided loads of a thread in flight.
    int found = 0;
    uint32_t low = 0xFFFFFFFFu, high = 0u;
    constexpr int kFlight = 8;
    for (int base = t; base < p.num_priors; base += kFlight * kClassThreads) {
      float s[kFlight];
#pragma unroll
      for (int u = 0; u < kFlight; ++u) {
        const int i = base + u * kClassThreads;
        if (i < p.num_priors) s[u] = scores[static_cast<size_t>(i) * p.num_classes];
      }
#pragma unroll
      for (int u = 0; u < kFlight; ++u) {
        const int i = base + u * kClassThreads;
        if (i >= p.num_priors) break;
        const bool pass = s[u] > p.confidence_threshold;
        const uint32_t key = pass ? descending_key(s[u]) : kNoKey;
        region[i] = key;
        if (pass) {
          ++found;
          low = min(low, key);
          high = max(high, key);
        }
      }
    }
    note_range(sh.select, low, high);
    found = __reduce_add_sync(0xffffffffu, found);
    if (lane == 0 && found) atomicAdd(&sh.num_cand, found);
  }
  __syncthreads();
  const int m = sh.num_cand;
  const int count = m < limit ? m : limit;
  auto each = [&](auto use) {
    for (int i = t; i < p.num_priors; i += kClassThreads) {
      const uint32_t key = region[i];
      if (key != kNoKey) use((static_cast<unsigned long long>(key) << 32) | static_cast<uint32_t>(i));
    }
  };
  unsigned long long threshold = kPadKey;
  if (m > limit) {
    // (a prior that does not pass sorts behind every one that does)
    auto fetch = [&](int i) { return (static_cast<unsigned long long>(region[i]) << 32) | static_cast<uint32_t>(i); };
    threshold = select_threshold(sh.select, each, fetch, p.num_priors, limit);
  }
  each([&](unsigned long long key) {
    if (key <= threshold) sel[atomicAdd(&sh.num_sel, 1)] = key;
  });
  __syncthreads();
  block_sort_keys(sel, padded);

  // Decode only the boxes that compete.
  const int loc_classes = p.share_location ? 1 : p.num_classes;
  const int loc_cls = p.share_location ? 0 : cls;
  const float* var = prior + static_cast<size_t>(p.num_priors) * 4;
  for (int i = t; i < count; i += kClassThreads) {
    const int pi = static_cast<int>(sel[i] & 0xFFFFFFFFull);
    const float* l = loc + ((static_cast<size_t>(image) * p.num_priors + pi) * loc_classes + loc_cls) * 4;
    const Box box = decode_box(p, prior + static_cast<size_t>(pi) * 4, var + static_cast<size_t>(pi) * 4, l);
    corners[i] = make_float4(box.xmin, box.ymin, box.xmax, box.ymax);
    sizes[i] = box.size;
  }
  __syncthreads();

  // Greedy NMS: candidate i is kept iff its overlap with every box kept so far
  // is <= the threshold.  With a fixed threshold (eta == 1, the usual case) the
  // overlaps do not depend on the walk: the whole block evaluates them into a bit matrix (word w of
  // column i, bit b: box 32 w + b < i would suppress box i), which takes the place of the score keys.
  // The kept set is then iterated from "all": a box stays unless a box that stays suppresses it.  Bit i
  // is final once those in front of it are, so this ends in the walk's own set, after as many rounds as
  // the longest chain of suppressions is long.
  // The bits of a list of up to 1024 have their place in the region if the limit is not above that; beyond it
  // the region was sized for the keys, which a short list's bits may still fit in.
  const int words = (count + 31) >> 5;
  const bool bits_fit = static_cast<size_t>(words) * count * sizeof(uint32_t) <= class_region_bytes(p.num_priors, limit);
  if (!(eta < 1.f) && words <= 32 && bits_fit) {
    uint32_t* suppress = region;
    const JaccardTest overlaps(p.nms_threshold);
    // A warp takes 32 rows x 32 columns at a time: lane = column, the rows are broadcasts.  (One thread
    // per word over the whole square, with five scalar loads per test: 70 k cycles for 400 boxes.)
    int column_block = 0, first_tile = 0;
    for (int tile = t >> 5; tile < words * (words + 1) / 2; tile += kClassThreads / 32) {
      while (tile > first_tile + column_block) first_tile += ++column_block;
      const int w = tile - first_tile;
      const int i = column_block * 32 + lane;
      const float4 cur = corners[min(i, count - 1)];
      const float cur_size = sizes[min(i, count - 1)];
      const int rows = min(32, count - w * 32);
      uint32_t bits = 0u, unsure = 0u;
#pragma unroll 4
      for (int r = 0; r < rows; ++r) {
        const int verdict = overlaps.quick(corners[w * 32 + r], sizes[w * 32 + r], cur, cur_size);
        bits |= static_cast<uint32_t>(verdict & 1) << r;
        unsure |= static_cast<uint32_t>(verdict >> 1) << r;
      }
      if (w == column_block) {      // only boxes in front suppress
        bits &= (1u << lane) - 1u;
        unsure &= (1u << lane) - 1u;
      }
      for (; unsure; unsure &= unsure - 1) {
        const int r = __ffs(unsure) - 1;
        if (jaccard(box_at(w * 32 + r), box_at(min(i, count - 1))) > p.nms_threshold) bits |= 1u << r;
      }
      if (i < count) suppress[w * count + i] = bits;
    }
    __syncthreads();
    // (count <= 1024: at most two groups of 32 columns per warp; `busy`: the words that hold anything)
    uint32_t busy[2] = {0u, 0u};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int g = (t >> 5) + u * (kClassThreads / 32), i = g * 32 + lane;
      if (g < words && i < count) {
        for (int w = 0; w <= g; ++w) busy[u] |= (suppress[w * count + i] != 0u ? 1u : 0u) << w;
      }
      const uint32_t all = __ballot_sync(0xffffffffu, i < count);
      if (lane == 0 && g < words) sh.keep[0][g] = all;
    }
    __syncthreads();
    for (int round = 0;; round ^= 1) {
      bool changed = false;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int g = (t >> 5) + u * (kClassThreads / 32), i = g * 32 + lane;
        if (g >= words) break;
        bool stays = i < count;
        for (uint32_t left = busy[u]; left && stays; left &= left - 1) {
          const int w = __ffs(left) - 1;
          stays = !(suppress[w * count + i] & sh.keep[round][w]);
        }
        const uint32_t next = __ballot_sync(0xffffffffu, stays);
        changed = changed || next != sh.keep[round][g];
        if (lane == 0) sh.keep[round ^ 1][g] = next;
      }
      if (!__syncthreads_or(changed)) break;
    }
  } else if (t < 32) {
    // Adaptive threshold (eta < 1) or a very long candidate list: one warp
    // compares each candidate with the kept list, 32 kept boxes at a time.
    float adaptive = p.nms_threshold;
    int nk = 0;
    for (int w = lane; w < 128; w += 32) sh.keep[0][w] = 0u;
    __syncwarp();
    for (int i = 0; i < count; ++i) {
      const Box cur = box_at(i);
      bool reject = false;
      for (int base = 0; base < nk && !reject; base += 32) {
        const int j = base + lane;
        const bool hit = j < nk && jaccard(cur, box_at(kept[j])) > adaptive;
        reject = __any_sync(0xffffffffu, hit);
      }
      if (!reject) {
        if (lane == 0) {
          kept[nk] = i;
          sh.keep[0][i >> 5] |= 1u << (i & 31);
        }
        ++nk;
        __syncwarp();
        if (eta < 1.f && adaptive > 0.5f) adaptive = fmul(adaptive, eta);
      }
    }
  }
  __syncthreads();
  Entry* out = ws.entries + (static_cast<size_t>(image) * p.num_classes + cls) * limit;
  for (int i = t; i < count; i += kClassThreads) {
    const uint32_t word = sh.keep[0][i >> 5];
    if (!((word >> (i & 31)) & 1u)) continue;
    int r = __popc(word & ((1u << (i & 31)) - 1u));
    for (int w = 0; w < (i >> 5); ++w) r += __popc(sh.keep[0][w]);
    const int pi = static_cast<int>(sel[i] & 0xFFFFFFFFull);
    Entry e;
    e.score = scores[static_cast<size_t>(pi) * p.num_classes];
    const float4 corner = corners[i];
    e.xmin = corner.x;
    e.ymin = corner.y;
    e.xmax = corner.z;
    e.ymax = corner.w;
    out[r] = e;
  }
  if (t == 0) {
    int total = 0;
    for (int w = 0; w < words; ++w) total += __popc(sh.keep[0][w]);
    *out_count = total;
  }
}

// ---------------------------------------------------------------- B. per image

constexpr int kImageThreads = 1024;

struct ImageShared {
  SelectShared select;
  int offsets[1025];   // first row of each class among the image's rows
  int selected[1024];  // rows kept per class
  int total;
};

// Running sums of values[0 .. n) (n <= 1024) into sums[0 .. n], by the whole block of 1024 threads.
__device__ void block_prefix_sum(SelectShared& sh, const int* values, int n, int* sums) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int own = t < n ? values[t] : 0;
  int incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) sh.warp_sum[warp] = incl;
  __syncthreads();
  int base = lane < warp ? sh.warp_sum[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
  if (t < n) sums[t] = base + incl - own;
  if (t == n - 1) sums[n] = base + incl;
  __syncthreads();
}

// `first_image`: the number of the grid's first image in the batch.
__global__ void __launch_bounds__(kImageThreads, 1)
detout_image_kernel(mcb200_detout_params p, Workspace ws, int first_image) {
  extern __shared__ __align__(16) unsigned char image_smem[];
  ImageShared& sh = *reinterpret_cast<ImageShared*>(image_smem);
  const int image = blockIdx.x;
  const int t = threadIdx.x;
  const int classes = p.num_classes;
  const int limit = ws.per_class;
  const int* counts = ws.class_count + static_cast<size_t>(image) * classes;
  const Entry* entries = ws.entries + static_cast<size_t>(image) * classes * limit;

  if (t == 0) {
    sh.select.low = 0xFFFFFFFFu;
    sh.select.high = 0u;
  }
  if (t < classes) sh.selected[t] = counts[t];
  __syncthreads();
  block_prefix_sum(sh.select, sh.selected, classes, sh.offsets);
  const int total = sh.offsets[classes];
  if (p.keep_top_k > -1 && total > p.keep_top_k) {
    // The keep_top_k best over all classes.  Key = (descending score, class * limit + rank); within a
    // class the entries are in descending score order, so the kept ones are a prefix of it.
    auto key_of = [&](int cell) { return make_key(entries[cell].score, static_cast<uint32_t>(cell)); };
    auto each = [&](auto use) {
      for (int cell = t; cell < classes * limit; cell += kImageThreads) {
        const int c = cell / limit;
        if (cell - c * limit < sh.offsets[c + 1] - sh.offsets[c]) use(key_of(cell));
      }
    };
    uint32_t low = 0xFFFFFFFFu, high = 0u;
    each([&](unsigned long long key) {
      low = min(low, static_cast<uint32_t>(key >> 32));
      high = max(high, static_cast<uint32_t>(key >> 32));
    });
    note_range(sh.select, low, high);
    __syncthreads();
    auto fetch = [&](int e) {   // e-th entry over the classes
      int c = 0;
      while (sh.offsets[c + 1] <= e) ++c;
      return key_of(c * limit + e - sh.offsets[c]);
    };
    unsigned long long threshold = 0ull;
    if (p.keep_top_k > 0) threshold = select_threshold(sh.select, each, fetch, total, p.keep_top_k);
    __syncthreads();
    if (t < classes) sh.selected[t] = 0;
    __syncthreads();
    if (p.keep_top_k > 0) {
      each([&](unsigned long long key) {
        if (key <= threshold) atomicAdd(&sh.selected[static_cast<uint32_t>(key) / limit], 1);
      });
    }
    __syncthreads();
    block_prefix_sum(sh.select, sh.selected, classes, sh.offsets);
  }
  if (t == 0) ws.image_count[image] = sh.offsets[classes];
  float* rows = ws.rows + static_cast<size_t>(image) * ws.max_rows * 7;
  for (int cell = t; cell < classes * limit; cell += kImageThreads) {
    const int c = cell / limit, j = cell - c * limit;
    if (j >= sh.selected[c]) continue;
    const Entry e = entries[cell];
    float* r = rows + static_cast<size_t>(sh.offsets[c] + j) * 7;
    r[0] = static_cast<float>(first_image + image);
    r[1] = static_cast<float>(c);
    r[2] = e.score;
    r[3] = e.xmin;
    r[4] = e.ymin;
    r[5] = e.xmax;
    r[6] = e.ymax;
  }
}

// ---------------------------------------------------------------- C. compaction

// One block per image: the block sums the counts of the images before its own
// (and of all images, for the total) and copies its rows behind them.
__global__ void __launch_bounds__(256)
detout_compact_kernel(Workspace ws, int batch, float* __restrict__ out, int* __restrict__ total_out) {
  __shared__ int sums[2];
  const int image = blockIdx.x;
  if (threadIdx.x == 0) sums[0] = sums[1] = 0;
  __syncthreads();
  int before = 0, all = 0;
  for (int i = threadIdx.x; i < batch; i += blockDim.x) {
    const int n = ws.image_count[i];
    all += n;
    if (i < image) before += n;
  }
  if (before) atomicAdd(&sums[0], before);
  if (all) atomicAdd(&sums[1], all);
  __syncthreads();
  const int first = sums[0], total = sums[1];
  const int n = ws.image_count[image];
  const float* rows = ws.rows + static_cast<size_t>(image) * ws.max_rows * 7;
  for (int i = threadIdx.x; i < n * 7; i += blockDim.x) out[static_cast<size_t>(first) * 7 + i] = rows[i];
  if (image == 0) {
    if (total == 0) {
      // No detection at all: one row per image, image id followed by -1.
      for (int i = threadIdx.x; i < batch * 7; i += blockDim.x) out[i] = (i % 7 == 0) ? static_cast<float>(i / 7) : -1.f;
    }
    if (threadIdx.x == 0) *total_out = total;
  }
}

int validate(const mcb200_detout_params* p, int batch) {
  if (!p || batch < 1) return -1;
  if (p->num_priors < 1 || p->num_classes < 1 || p->num_classes > 1024 || p->code_type < 1 || p->code_type > 3)
    return -2;
  if (batch > 65535) return -3;
  if (!(p->eta > 0.f) || p->eta > 1.f) return -8;
  const int limit = per_class_limit(*p);
  if (det::next_pow2(limit) > 4096) return -4;
  return 0;
}

size_t class_kernel_smem(const mcb200_detout_params& p, int padded) {
  return ((sizeof(ClassShared) + 15) & ~static_cast<size_t>(15)) + static_cast<size_t>(padded) * (8 + sizeof(float4) + sizeof(float) + sizeof(int)) +
         class_region_bytes(p.num_priors, per_class_limit(p));
}

}  // namespace
}  // namespace mcb200

using namespace mcb200;

extern "C" size_t mcb200_detout_workspace_bytes(const mcb200_detout_params* p, int batch) {
  if (validate(p, batch) != 0) return 0;
  return carve(*p, batch, nullptr, nullptr);
}

extern "C" int mcb200_detout_max_rows_per_image(const mcb200_detout_params* p) {
  if (validate(p, 1) != 0) return -1;
  const int rows = max_rows(*p);
  return rows > 1 ? rows : 1;
}

// Opts a kernel into the shared memory it needs, once per device and size.
static cudaError_t allow_shared(const void* kernel, size_t bytes, size_t* configured) {
  static std::mutex mu;   // nets on several host threads may make their first call together
  std::lock_guard<std::mutex> lock(mu);
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || configured[dev] >= bytes) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e == cudaSuccess) configured[dev] = bytes;
  return e;
}

extern "C" int mcb200_detout_part(const mcb200_detout_params* p, int batch, int first_image, int images, const float* loc,
                                  const float* conf, const float* prior, void* workspace, void* stream) {
  const int rc = validate(p, batch);
  if (rc != 0) return rc;
  if (!loc || !conf || !prior || !workspace) return -5;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return -6;
  if (first_image < 0 || images < 1 || first_image + images > batch) return -9;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Workspace ws;
  carve(*p, batch, static_cast<char*>(workspace), &ws);
  ws.entries += static_cast<size_t>(first_image) * p->num_classes * ws.per_class;
  ws.class_count += static_cast<size_t>(first_image) * p->num_classes;
  ws.rows += static_cast<size_t>(first_image) * ws.max_rows * 7;
  ws.image_count += first_image;
  // (Two keys at least: the boxes behind them are read 16 bytes at a time.)
  const int padded = ws.per_class > 1 ? det::next_pow2(ws.per_class) : 2;
  const size_t smem = class_kernel_smem(*p, padded);
  if (smem > 220 * 1024) return -7;
  static size_t class_configured[64], image_configured[64];
  cudaError_t e = allow_shared(reinterpret_cast<const void*>(detout_class_kernel), smem, class_configured);
  if (e != cudaSuccess) return static_cast<int>(e);
  e = allow_shared(reinterpret_cast<const void*>(detout_image_kernel), sizeof(ImageShared), image_configured);
  if (e != cudaSuccess) return static_cast<int>(e);
  detout_class_kernel<<<dim3(p->num_classes, images), kClassThreads, smem, st>>>(loc, conf, prior, *p, ws, padded, p->eta);
  count_launch();
  detout_image_kernel<<<images, kImageThreads, sizeof(ImageShared), st>>>(*p, ws, first_image);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_detout_finish(const mcb200_detout_params* p, int batch, void* workspace, float* out, int* total,
                                    void* stream) {
  const int rc = validate(p, batch);
  if (rc != 0) return rc;
  if (!workspace || !out || !total) return -5;
  Workspace ws;
  carve(*p, batch, static_cast<char*>(workspace), &ws);
  detout_compact_kernel<<<batch, 256, 0, static_cast<cudaStream_t>(stream)>>>(ws, batch, out, total);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_detout_forward(const mcb200_detout_params* p, int batch, const float* loc, const float* conf,
                                     const float* prior, void* workspace, float* out, int* total, void* stream) {
  if (!out || !total) return p ? -5 : -1;
  const int rc = mcb200_detout_part(p, batch, 0, batch, loc, conf, prior, workspace, stream);
  return rc != 0 ? rc : mcb200_detout_finish(p, batch, workspace, out, total, stream);
}
