// 3 x 3 convolution, stride 1, padding 1, of at most 64 to at most 64 channels, on wide maps: the tensor-core form in
// which every input row is loaded once.
//
// The general kernel (conv_tc.cu) multiplies such a layer in tiles of 64 columns: an MMA of 128 x 64 x 8 reads six
// kilobytes of operands for what is 32 cycles of arithmetic, an input row is fetched for each of the three
// filter rows, and the loop waits for it (64 -> 64 channels at 300 x 300, batch 32: 397 TFLOP/s of the tensor
// pipe's 1107).  Here a CTA marches down the image.  An input row contributes to three output rows, whose
// accumulators of 64 columns lie side by side in tensor memory: with the weights of the three filter rows stacked to
// 192 rows, one MMA of 128 x 192 x 8 adds to all three.  That is ten kilobytes of operands in
// 96 cycles, which the shared-memory port (128 bytes per cycle) delivers at the pipe's full rate.  All weights stay in shared
// memory (147 KB in fp32); what streams are the input rows, 32 KB per 2304 cycles.
//
// The 128 rows of an MMA are two slabs of 64 neighbouring pixels (62 outputs and the filter's overhang).  A column is a
// segment of at most 62 pixels of the rows of one image, with a row of padding above and below; all columns, one behind the
// other, are one tall image that is cut into equal runs, one per slab: every CTA has the same number of rows, and a
// run that crosses from one column into the next only computes two rows that nobody stores.  Output row u
// accumulates in slot u mod 8 of tensor memory, so the epilogue may lag six rows behind.
//   warp 0     one thread loads the weights, then a row of each slab per step (tiled tensor map, zero fill outside
//              the image is the padding)
//   warp 1     one thread issues the MMAs: taps of a filter row read the same pixels one further down, as
//              in the general kernel's halo mode
//   warps 2-9  per-channel scale / shift, activation, stores straight from the registers
// Every wait is bounded; a timed-out wait raises an abort flag and *status.
//
// A 2 x 2 max pooling of stride 2 behind the layer is taken in the epilogue: neighbouring rows are neighbouring
// accumulators of the same lanes, and the unpooled map, four times the result, is neither written nor read.
//
// The sum over K runs over filter rows, then channel blocks, then taps, whatever the batch.
// Measured: 64 -> 64 channels at 300 x 300, batch 32, with the pooling behind it 565 + 130 -> 301 us; at 56 x 56, batch 64,
// 49.7 -> 34.  A row takes 3400 cycles where its MMAs need 2304.  In a run of four rows (56 x 56, batch 16, 18 us) the tensor
// pipe is active 57 % of an SM's cycles, 72 % on the busiest; its shared-memory reads take a third of theirs.
// Arithmetic replaced: mini-caffe's im2col + SGEMM + bias (src/layers/base_conv_layer.cpp:254-278).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "../../../include/mcb200_kernels.h"
#include "kernel_timer.h"
#include "launch_count.h"
#include "sm100.cuh"

namespace mcb200 {

// The convolution kernels' common settings (conv_tc.cu): bound of their waits, and the one-shot test hook.
long long conv_wait_limit();
int conv_take_drop_hook();

namespace {

using namespace sm100;

constexpr int kSlab = 64;            // MMA rows of a slab
constexpr int kSlabOutputs = 62;     // of which a filter three pixels wide leaves these
constexpr int kFewestRows = 3;       // of a slab
constexpr int kSlots = 8;            // accumulators of 64 columns: all of tensor memory
constexpr int kColumns = 64;
constexpr int kStageBytes = 2 * kSlab * 128;            // a row of both slabs, one channel block
constexpr int kWeightTile = 3 * kColumns * 128;         // one tap column and channel block, three filter rows
constexpr int kMaxStages = 8;
constexpr int kEpilogueWarps = 8;
constexpr int kFirstEpilogueWarp = 2;
constexpr int kThreads = (kFirstEpilogueWarp + kEpilogueWarps) * 32;
constexpr int kSharedLimit = 232448;

struct MarchArgs {
  void* out;
  int out_ld, out_half, vec;
  int cout, h, w;
  int segments, segment_w;   // columns of an image, outputs of a column's row
  int column_h, pad_top;     // rows of a column, and of padding above the image
  int total, run;            // rows of all columns, and of a slab's run
  mcb200_epilogue ep;
  int stages;
  int constants_settled;
  int drop_last_load;        // test hook, see mcb200_conv_test_drop_weight_load
  int* status;
  long long wait_limit;
};

// A slab's place in the tall image: column and image row (above 0 and below h - 1: padding).
struct Place {
  int column, y;
  __device__ __forceinline__ void set(int row, const MarchArgs& a) {
    column = row < 0 ? 0 : row / a.column_h;   // (the row in front of the first column's padding: zeros as well)
    y = row - column * a.column_h - a.pad_top;
  }
  __device__ __forceinline__ void next(const MarchArgs& a) {
    if (++y == a.column_h - a.pad_top) {
      y = -a.pad_top;
      ++column;
    }
  }
};

template <int kValue>
struct Wrap {
  static constexpr int value = kValue;
};

template <int kBlocks, bool kHalf, bool kPool>
__global__ void __launch_bounds__(kThreads, 1)
conv_march_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const MarchArgs args) {
  constexpr int kElems = kHalf ? 64 : 32;   // channels of a block
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages];
  __shared__ uint64_t row_full[kSlots], row_empty[kSlots];
  __shared__ uint64_t weights_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const uint32_t raw = smem_addr(smem_raw);
  uint8_t* ring = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  const int stages = args.stages;
  uint8_t* weights = ring + stages * kStageBytes;   // behind the ring: the taps of the last stage's last pixels read on into it
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long wait_limit = args.wait_limit;
  const int steps = args.run + 2;                   // input rows of a run

  {
    const int t = static_cast<int>(threadIdx.x);
    if (t == 0) abort_flag = 0;
    if (t < stages) {
      mbar_init(&full_bar[t], 1);
      mbar_init(&empty_bar[t], 1);
    } else if (t >= 32 && t < 32 + kSlots) {
      mbar_init(&row_full[t - 32], 1);
      mbar_init(&row_empty[t - 32], kEpilogueWarps);
    } else if (t == 64) {
      mbar_init(&weights_bar, 1);
    } else if (t == 65) {
      tma_prefetch_descriptor(&map_a);
      tma_prefetch_descriptor(&map_b);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  volatile int* abort = &abort_flag;
  grid_launch_dependents();
  if (args.constants_settled == 0 || warp == 1) grid_dependency_wait();

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(&weights_bar, 3 * kBlocks * kWeightTile);
      for (int i = 0; i < 3 * kBlocks; ++i) tma_load_2d(&map_b, &weights_bar, weights + i * kWeightTile, i * kElems, 0);
      if (args.constants_settled != 0) grid_dependency_wait();
      Place place[2];
      for (int i = 0; i < 2; ++i) place[i].set((static_cast<int>(blockIdx.x) * 2 + i) * args.run - 1, args);
      int stage = 0, issued = 0;
      uint32_t parity = 0;
      bool alive = true;
      for (int step = 0; step < steps && alive; ++step) {
        int x[2], n[2];
        for (int i = 0; i < 2; ++i) {
          n[i] = place[i].column / args.segments;   // past the last image: zeros, which nobody stores
          x[i] = (place[i].column - n[i] * args.segments) * args.segment_w - 1;
        }
        for (int block = 0; block < kBlocks; ++block) {
          if (!mbar_wait_bounded(&empty_bar[stage], parity ^ 1u, abort, wait_limit)) {
            alive = false;
            break;
          }
          if (args.drop_last_load && step + 1 == steps && block + 1 == kBlocks) {
            alive = false;   // nothing arrives on this stage's barrier: every role's wait on it is bounded
            break;
          }
          mbar_expect_tx(&full_bar[stage], kStageBytes);
          uint8_t* dst = ring + stage * kStageBytes;
          for (int i = 0; i < 2; ++i)
            tma_load_4d(&map_a, &full_bar[stage], dst + i * kSlab * 128, block * kElems, x[i], place[i].y, n[i]);
          ++issued;
          if (++stage == stages) {
            stage = 0;
            parity ^= 1u;
          }
        }
        place[0].next(args);
        place[1].next(args);
      }
      // Copies in flight land before the CTA gives its shared memory back (bounded).
      if (*abort) {
        for (int j = issued > stages ? issued - stages : 0; j < issued; ++j) {
          const long long start = clock64();
          while (!mbar_try_wait(&full_bar[j % stages], static_cast<uint32_t>(j / stages) & 1u)) {
            if (clock64() - start > wait_limit / 8) break;
          }
        }
        const long long start = clock64();
        while (!mbar_try_wait(&weights_bar, 0u)) {
          if (clock64() - start > wait_limit / 8) break;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc1 = kHalf ? umma_idesc_bf16(128, 64) : umma_idesc_tf32(128, 64);
      constexpr uint32_t idesc2 = kHalf ? umma_idesc_bf16(128, 128) : umma_idesc_tf32(128, 128);
      constexpr uint32_t idesc3 = kHalf ? umma_idesc_bf16(128, 192) : umma_idesc_tf32(128, 192);
      auto mma = [&](uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
        if (kHalf) {
          umma_bf16(d, da, db, idesc, accumulate);
        } else {
          umma_tf32(d, da, db, idesc, accumulate);
        }
      };
      constexpr uint64_t kRow = kColumns * 128 / 16;       // from one filter row's weights to the next, in descriptor units
      constexpr uint64_t kTile = kWeightTile / 16;
      const uint32_t ring_addr = smem_addr(ring);
      const uint64_t weights_desc = umma_desc_k_sw128(smem_addr(weights));
      int stage = 0;
      uint32_t parity = 0;
      // One input row.  kWrap: how its three output rows lie in the eight slots: side by side from `first` on, or with
      // the last one, or the last two, in the first slots.  Straight-line code: with the cases decided per
      // MMA the issuing thread, not the tensor pipe, set the pace.
      auto issue_row = [&](auto wrap_tag, uint32_t first) {
        constexpr int kWrap = decltype(wrap_tag)::value;
#pragma unroll
        for (int block = 0; block < kBlocks; ++block) {
          if (!mbar_wait_bounded(&full_bar[stage], parity, abort, wait_limit)) return false;
          tc_fence_after_sync();
          const uint64_t stage_desc = umma_desc_k_sw128(ring_addr + static_cast<uint32_t>(stage * kStageBytes));
#pragma unroll
          for (int s = 0; s < 3; ++s) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint64_t a = stage_desc + s * 8 + 2 * kk;     // tap s: a pixel, 128 bytes, further down
              const uint64_t b = weights_desc + (s * kBlocks + block) * kTile + 2 * kk;
              const bool fresh = block == 0 && s == 0 && kk == 0;   // the new output row's first contribution
              if (kWrap == 0 && !fresh) {
                mma(first, a, b, idesc3, 1u);
              } else if (kWrap <= 1) {
                mma(first, a, b, idesc2, 1u);
                mma(kWrap == 0 ? first + 2 * kColumns : tmem, a, b + 2 * kRow, idesc1, fresh ? 0u : 1u);
              } else {
                mma(first, a, b, idesc1, 1u);
                if (fresh) {
                  mma(tmem, a, b + kRow, idesc1, 1u);
                  mma(tmem + kColumns, a, b + 2 * kRow, idesc1, 0u);
                } else {
                  mma(tmem, a, b + kRow, idesc2, 1u);
                }
              }
            }
          }
          umma_commit(&empty_bar[stage]);
          if (++stage == stages) {
            stage = 0;
            parity ^= 1u;
          }
        }
        return true;
      };
      bool alive = mbar_wait_bounded(&weights_bar, 0u, abort, wait_limit);
      for (int step = 0; step < steps && alive; ++step) {
        // This input row is the last filter row's of output step - 2, the middle one's of step - 1 and the first
        // one's of `step`, whose slot the epilogue must have drained.
        if (!mbar_wait_bounded(&row_empty[step & 7], (static_cast<uint32_t>(step >> 3) & 1u) ^ 1u, abort, wait_limit)) break;
        tc_fence_after_sync();
        const int slot = (step - 2) & 7;
        const uint32_t first = tmem + static_cast<uint32_t>(slot * kColumns);
        alive = slot <= 5 ? issue_row(Wrap<0>(), first) : slot == 6 ? issue_row(Wrap<1>(), first) : issue_row(Wrap<2>(), first);
        if (alive && step >= 2) umma_commit(&row_full[slot]);
      }
    }
  } else {
    const int ew = warp - kFirstEpilogueWarp;
    const int quad = warp & 3, half = ew >> 2;     // tensor-memory lanes [32 quad, + 32), columns [32 half, + 32)
    const int col_in = 2 * (lane & 3), row_in = lane >> 2;
    const mcb200_epilogue& ep = args.ep;
    float2 scale[4], shift[4], slope[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float v[3][2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = half * 32 + 8 * j + col_in + e;
        const bool in = c < args.cout;
        v[0][e] = in && ep.scale ? __ldg(ep.scale + c) : 1.f;
        v[1][e] = in && ep.shift ? __ldg(ep.shift + c) : 0.f;
        v[2][e] = ep.act == 2 ? (in && ep.prelu ? __ldg(ep.prelu + (ep.prelu_shared ? 0 : c)) : 0.f) : ep.slope;
      }
      scale[j] = make_float2(v[0][0], v[0][1]);
      shift[j] = make_float2(v[1][0], v[1][1]);
      slope[j] = make_float2(v[2][0], v[2][1]);
    }
    if (args.constants_settled != 0) grid_dependency_wait();
    const int act_mode = ep.act == 0 ? 0 : ((ep.act == 1 && ep.slope == 0.f) ? 1 : 2);
    const int first = (static_cast<int>(blockIdx.x) * 2 + (quad >> 1)) * args.run;   // of this warp's slab
    const int pixel0 = (quad & 1) * 32 + row_in;                                      // first of this lane's pixels, 8 apart
    Place place;
    place.set(first, args);
    // Waits for output row u of the run and reads this warp's part of it.
    auto read_row = [&](int u, uint32_t (&acc)[2][16]) {
      const int slot = u & 7;
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&row_full[slot], static_cast<uint32_t>(u >> 3) & 1u, abort, wait_limit))) return false;
      tc_fence_after_sync();
      const uint32_t at = tmem + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(slot * kColumns + half * 32);
      tmem_load_16x256<4>(at, acc[0]);
      tmem_load_16x256<4>(at + (16u << 16), acc[1]);
      tmem_load_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&row_empty[slot]);
      return true;
    };
    auto finish = [&](uint32_t (&acc)[2][16]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t& cell = acc[i >> 1][4 * j + 2 * (i & 1) + e];
            float v = fmaf(__uint_as_float(cell), e ? scale[j].y : scale[j].x, e ? shift[j].y : shift[j].x);
            if (act_mode == 1) {
              v = fmaxf(v, 0.f);
            } else if (act_mode == 2) {
              v = v > 0.f ? v : v * (e ? slope[j].y : slope[j].x);
            }
            if (ep.round_tf32) v = round_to_tf32(v);
            cell = __float_as_uint(v);
          }
        }
      }
    };
    // Row set i goes to output row `row` + its pixel (all lanes call it: bfloat16 columns change lanes).
    auto store = [&](const uint32_t (&acc)[2][16], int i, bool there, size_t row) {
      const size_t to = row * args.out_ld + half * 32;
      uint32_t w[4][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w[j][0] = acc[i >> 1][4 * j + 2 * (i & 1)];
        w[j][1] = acc[i >> 1][4 * j + 2 * (i & 1) + 1];
      }
      if (args.out_half && args.vec) {
        uint32_t packed[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) packed[j] = pack_bf16x2(__uint_as_float(w[j][0]), __uint_as_float(w[j][1]));
        quad_transpose(packed, lane & 3);
        const int c = 8 * (lane & 3);
        if (there && half * 32 + c < args.cout)
          *reinterpret_cast<uint4*>(static_cast<uint16_t*>(args.out) + to + c) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        return;
      }
      if (!there) return;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = 8 * j + col_in;
        const float v0 = __uint_as_float(w[j][0]), v1 = __uint_as_float(w[j][1]);
        if (half * 32 + c >= args.cout) continue;
        if (args.vec) {
          *reinterpret_cast<float2*>(static_cast<float*>(args.out) + to + c) = make_float2(v0, v1);
        } else if (args.out_half) {
          uint16_t* dst = static_cast<uint16_t*>(args.out) + to + c;
          dst[0] = static_cast<uint16_t>(pack_bf16x2(v0, 0.f));
          if (half * 32 + c + 1 < args.cout) dst[1] = static_cast<uint16_t>(pack_bf16x2(v1, 0.f));
        } else {
          float* dst = static_cast<float*>(args.out) + to + c;
          dst[0] = v0;
          if (half * 32 + c + 1 < args.cout) dst[1] = v1;
        }
      }
    };
    for (int u = 0; u < args.run; u += kPool ? 2 : 1) {
      uint32_t acc[2][16], below[2][16];
      if (!read_row(u, acc)) break;
      if (kPool && !read_row(u + 1, below)) break;
      const int n = place.column / args.segments, y = place.y;
      const int x0 = (place.column - n * args.segments) * args.segment_w;
      const int pixels = first + u < args.total && y >= 0 && y < args.h ? min(args.segment_w, args.w - x0) : 0;
      place.next(args);
      if (kPool) place.next(args);
      if (pixels == 0) continue;
      finish(acc);
      if (!kPool) {
        const size_t row = (static_cast<size_t>(n) * args.h + y) * args.w + x0;
#pragma unroll
        for (int i = 0; i < 4; ++i) store(acc, i, pixel0 + 8 * i < pixels, row + pixel0 + 8 * i);
        continue;
      }
      // 2 x 2 maxima: runs begin at even rows and segments at even pixels, so a window is two rows of one
      // run and two neighbouring pixels, four lanes apart.  Windows at the last row or pixel may be cut.
      finish(below);
      // Cells that a cut window lacks count as the lowest value of the result's type, whole windows as they are
      // (all -infinity, all NaN): the pooling kernels' rules, whose general one, for columns that are no multiple of four,
      // starts every window at the lowest value.  (fmaxf with NaN is its other operand.)
      const bool two_rows = y + 1 < args.h;
      const float lowest = args.out_half ? __uint_as_float(0xff7f0000u) : -3.402823466e+38f;
      const size_t row = (static_cast<size_t>(n) * ((args.h + 1) >> 1) + (y >> 1)) * ((args.w + 1) >> 1);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pixel = pixel0 + 8 * i;
        const bool two_pixels = (pixel & 1) != 0 || pixel + 1 < pixels;
        const float least = two_rows && two_pixels && (args.cout & 3) == 0 ? __uint_as_float(0x7fffffffu) : lowest;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          uint32_t& cell = acc[i >> 1][4 * (k >> 1) + 2 * (i & 1) + (k & 1)];
          float v = fmaxf(least, __uint_as_float(cell));
          if (two_rows) v = fmaxf(v, __uint_as_float(below[i >> 1][4 * (k >> 1) + 2 * (i & 1) + (k & 1)]));
          const float beside = __shfl_xor_sync(0xffffffffu, v, 4);
          cell = __float_as_uint(two_pixels ? fmaxf(v, beside) : v);
        }
        store(acc, i, (pixel & 1) == 0 && pixel < pixels, row + ((x0 + pixel) >> 1));
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && abort_flag && args.status) *static_cast<volatile int*>(args.status) = 1;
}

// [cout][c][3][3] -> [filter row 2, 1, 0][64 output channels][tap column][blocks x 32 (64) channels], zero beyond both counts.
template <bool kHalf>
__global__ void pack_march_weights_kernel(const float* __restrict__ w, void* __restrict__ packed, int cout, int c, int c_pad) {
  const int total = 3 * kColumns * 3 * c_pad;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int cc = i % c_pad, s = i / c_pad % 3;
    const int row = i / (3 * c_pad);
    const int co = row % kColumns, r = 2 - row / kColumns;
    const float v = cc < c && co < cout ? w[(static_cast<size_t>(co) * c + cc) * 9 + r * 3 + s] : 0.f;
    if (kHalf) {
      static_cast<uint16_t*>(packed)[i] = static_cast<uint16_t>(pack_bf16x2(v, 0.f));
    } else {
      static_cast<float*>(packed)[i] = round_to_tf32(v);
    }
  }
}

int blocks_of(const mcb200_conv_shape& s, bool half) { return (s.c + (half ? 63 : 31)) / (half ? 64 : 32); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

template <int kBlocks, bool kHalf, bool kPool>
cudaError_t launch(const mcb200_march_plan* plan, MarchArgs args, cudaStream_t stream) {
  auto kernel = conv_march_kernel<kBlocks, kHalf, kPool>;
  constexpr int kWeights = 3 * kBlocks * kWeightTile;
  static std::mutex mu;
  static bool configured[64] = {false};
  static int sms[64] = {0}, limit = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (limit == 0) {
      cudaFuncAttributes attr;
      cudaError_t e = cudaFuncGetAttributes(&attr, kernel);
      if (e != cudaSuccess) return e;
      limit = kSharedLimit - static_cast<int>(attr.sharedSizeBytes);
    }
    if (!configured[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
      if (e != cudaSuccess) return e;
      if (cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms[dev] < 1) sms[dev] = 148;
      configured[dev] = true;
    }
  }
  int stages = (limit - 1024 - kWeights) / kStageBytes;
  if (stages > kMaxStages) stages = kMaxStages;
  if (stages < 2) return cudaErrorInvalidConfiguration;
  args.stages = stages;
  const long long slabs = 2LL * sms[dev];
  args.run = static_cast<int>((args.total + slabs - 1) / slabs);
  if (kPool) args.run += args.run & 1;
  const int grid = (args.total + 2 * args.run - 1) / (2 * args.run);
  TimedLaunch timed(stream);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = static_cast<size_t>(stages * kStageBytes + kWeights + 1024);   // + alignment slack
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, *reinterpret_cast<const CUtensorMap*>(plan->tma_a),
                                           *reinterpret_cast<const CUtensorMap*>(plan->tma_b), args);
  count_launch();
  return e;
}

}  // namespace
}  // namespace mcb200

using namespace mcb200;

// What the kernel takes: rows that fill three quarters of their slabs.
extern "C" int mcb200_conv_march_supported(const mcb200_conv_shape* s, int operands_bf16) {
  if (!s || s->group != 1 || s->kh != 3 || s->kw != 3 || s->stride_h != 1 || s->stride_w != 1 || s->pad_h != 1 || s->pad_w != 1 ||
      s->dil_h != 1 || s->dil_w != 1)
    return 0;
  if (s->c <= 32 || s->c > 64 || s->cout <= 32 || s->cout > kColumns || s->c % (operands_bf16 ? 8 : 4) != 0) return 0;
  if (s->h < 1 || s->w < 1) return 0;
  const int segments = (s->w + kSlabOutputs - 1) / kSlabOutputs;
  return 4LL * s->w >= 3LL * kSlab * segments;
}

// And whether there are at least kFewestRows rows for each slab: a run loads two rows more than it finishes.  (The
// general kernel's halo mode adds the same products in the same order: the bits do not depend on the choice.)
// At 56 x 56 one image (a row per slab) takes 14.8 us here and 10.6 there; sixteen in bfloat16 (four rows) 14.8 both ways
// in runs of one launch at a time, and 3 us less per pass here.
extern "C" int mcb200_conv_march_pays(const mcb200_conv_shape* s, int operands_bf16) {
  return mcb200_conv_march_supported(s, operands_bf16) && mcb200_conv_march_rows_per_slab(s) >= kFewestRows;
}

extern "C" int mcb200_conv_march_rows_per_slab(const mcb200_conv_shape* s) {
  if (!s || s->n < 0 || s->h < 1 || s->w < 1) return 0;
  const int segments = (s->w + kSlabOutputs - 1) / kSlabOutputs;
  const long long rows = static_cast<long long>(s->n) * segments * (s->h + 2LL) / (2 * 148);
  return rows < 0x7fffffff ? static_cast<int>(rows) : 0x7fffffff;
}

extern "C" size_t mcb200_conv_march_packed_weight_bytes(const mcb200_conv_shape* s, int operands_bf16) {
  return s ? static_cast<size_t>(3 * blocks_of(*s, operands_bf16 != 0)) * kWeightTile : 0;
}

extern "C" int mcb200_conv_march_pack_weights(const mcb200_conv_shape* s, int operands_bf16, const float* w_oihw, void* packed,
                                              void* stream) {
  if (!w_oihw || !packed || !mcb200_conv_march_supported(s, operands_bf16)) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (operands_bf16) {
    pack_march_weights_kernel<true><<<148, 256, 0, st>>>(w_oihw, packed, s->cout, s->c, blocks_of(*s, true) * 64);
  } else {
    pack_march_weights_kernel<false><<<148, 256, 0, st>>>(w_oihw, packed, s->cout, s->c, blocks_of(*s, false) * 32);
  }
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_conv_march_plan(const mcb200_conv_shape* s, int operands_bf16, const void* in, const void* packed_w,
                                      int pool, mcb200_march_plan* plan) {
  const bool half = operands_bf16 != 0;
  if (!in || !packed_w || !plan || !mcb200_conv_march_supported(s, operands_bf16)) return -1;
  if (s->c_stride < s->c || (s->c_stride & (half ? 7 : 3)) != 0) return -2;
  if ((reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(packed_w) & 15)) return -3;
  EncodeTiledFn encode = encode_tiled();
  if (!encode) return -5;
  plan->shape = *s;
  if (mcb200_conv_out_shape(&plan->shape) != 0) return -6;
  const int segments = (s->w + kSlabOutputs - 1) / kSlabOutputs;
  // Pooled: an even number of rows above the image and in a column.
  plan->pool = pool ? 1 : 0;
  plan->pad_top = pool ? 2 : 1;
  plan->column_h = pool ? (s->h + 4) / 2 * 2 : s->h + 2;
  const long long total = static_cast<long long>(s->n) * segments * plan->column_h;
  const long long pixels = static_cast<long long>(s->n) * s->h * s->w;
  if (s->n < 1 || total > 0x3fffffff || pixels > 0x7fffffffLL) return -7;
  plan->operand_bf16 = half ? 1 : 0;
  plan->segments = segments;
  plan->segment_w = (s->w + segments - 1) / segments;
  if (pool) plan->segment_w += plan->segment_w & 1;
  plan->total = static_cast<int>(total);
  const CUtensorMapDataType type = half ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const cuuint32_t elems = half ? 64 : 32;
  const cuuint64_t es = half ? 2 : 4, pix = static_cast<cuuint64_t>(s->c_stride) * es;
  const cuuint32_t ones[4] = {1, 1, 1, 1};
  {
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(s->c), static_cast<cuuint64_t>(s->w), static_cast<cuuint64_t>(s->h),
                                static_cast<cuuint64_t>(s->n)};
    const cuuint64_t strides[3] = {pix, pix * s->w, pix * s->w * s->h};
    const cuuint32_t box[4] = {elems, kSlab, 1, 1};
    const CUresult r = encode(reinterpret_cast<CUtensorMap*>(plan->tma_a), type, 4, const_cast<void*>(in), dims, strides, box, ones,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -100 - static_cast<int>(r);
  }
  {
    const cuuint64_t cols = static_cast<cuuint64_t>(3 * blocks_of(*s, half)) * elems;
    const cuuint64_t dims[2] = {cols, 3 * kColumns};
    const cuuint64_t strides[1] = {cols * es};
    const cuuint32_t box[2] = {elems, 3 * kColumns};
    const CUresult r = encode(reinterpret_cast<CUtensorMap*>(plan->tma_b), type, 2, const_cast<void*>(packed_w), dims, strides, box,
                              ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -200 - static_cast<int>(r);
  }
  return 0;
}

extern "C" int mcb200_conv_march_launch(const mcb200_march_plan* plan, void* out, int out_is_bf16, int out_ld,
                                        const mcb200_epilogue* ep, int flags, int* status, void* stream) {
  if (!plan || !out || !ep || ep->residual || out_ld < plan->shape.cout || (ep->act == 2 && !ep->prelu)) return -1;
  const bool half = plan->operand_bf16 != 0;
  MarchArgs a;
  a.out = out;
  a.out_ld = out_ld;
  a.out_half = out_is_bf16 ? 1 : 0;
  const int wide = a.out_half ? 8 : 2;   // columns of a wide store: two fp32, eight bfloat16
  a.vec = out_ld % wide == 0 && plan->shape.cout % wide == 0 && (reinterpret_cast<uintptr_t>(out) & (a.out_half ? 15 : 7)) == 0;
  a.cout = plan->shape.cout;
  a.h = plan->shape.h;
  a.w = plan->shape.w;
  a.segments = plan->segments;
  a.segment_w = plan->segment_w;
  a.column_h = plan->column_h;
  a.pad_top = plan->pad_top;
  a.total = plan->total;
  a.ep = *ep;
  a.constants_settled = (flags & MCB200_CONV_CONSTANTS_SETTLED) ? 1 : 0;
  a.status = status;
  a.wait_limit = conv_wait_limit();
  a.drop_last_load = conv_take_drop_hook();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return static_cast<int>(plan->pool ? (half ? launch<1, true, true>(plan, a, st) : launch<2, false, true>(plan, a, st))
                                     : (half ? launch<1, true, false>(plan, a, st) : launch<2, false, false>(plan, a, st)));
}
