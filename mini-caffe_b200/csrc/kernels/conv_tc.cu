// Convolution / InnerProduct as an implicit GEMM on the Blackwell tensor cores.
//
//   D[m, co] = sum over taps (r, s) and channels c of  X[pixel(m) + (r, s), c] * W[co, r, s, c]
//
// m runs over the N*Ho*Wo output pixels of a channels-last activation tensor.
// One CTA computes 128 x BN tiles of D, one after the other (persistent):
//   warp 0   one elected thread issues the activation loads.  The tile (128
//            pixels x 32 channels of one filter tap) comes through an
//            im2col-mode tensor map, so the hardware walks the output pixels
//            across image rows and images and zero-fills the padding.
//   warp 2   one elected thread issues the weight loads (BN x 32, tiled map).
//            Both operands land in shared memory 128-byte swizzled, K-major.
//            Two issuing threads because a single thread's loop (wait, arm the
//            barrier, issue) costs a few hundred cycles per k-iteration, which
//            is as long as the copy itself takes.
//   warp 1   one thread issues tcgen05.mma kind::tf32 (M=128, N=BN, K=8), four per
//            stage, accumulating in tensor memory; tcgen05.commit hands each
//            shared-memory stage back to the producers.
//   warps 3-10 read the accumulator out of tensor memory (tcgen05.ld), apply
//            the fused tail (per-channel scale/shift, residual add, ReLU or
//            PReLU) and store channels-last.  Two warps share each 32-lane
//            quadrant of tensor memory and take alternate chunks of columns.  Results go
//            straight from registers to memory, or, where many tiles keep HBM busy, through
//            swizzled 32 x 32 sub-tiles in shared memory and out as TMA tile stores, a
//            residual the same way in (see staged_epilogue).
// Every barrier wait is bounded; a timed-out wait raises an abort flag, the
// roles drain, tensor memory is freed and *status is set.
//
// Arithmetic replaced: mini-caffe's per-image im2col + SGEMM + bias GEMM
// (src/layers/base_conv_layer.cpp:254-278, src/util/im2col.cpp:19-55).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <stdlib.h>

#include <algorithm>
#include <mutex>

#include "../../../include/mcb200_kernels.h"
#include "kernel_timer.h"
#include "launch_count.h"
#include "sm100.cuh"

namespace mcb200 {
namespace {

using namespace sm100;

constexpr int kBlockM = 128;
constexpr int kSmallM = 64;                            // M tile of a launch too small for the chip, see small_tiles
constexpr int kBlockK = 32;                            // fp32 elements = one 128-byte swizzle row
constexpr int kBlockKHalf = 64;                        // bfloat16 elements of the same 128 bytes
constexpr int kMmaPerBlock = 4;                        // 32-byte K steps of a swizzle row (K = 8 tf32 / 16 bf16)
constexpr int kTileABytes = kBlockM * kBlockK * 4;     // 16 KiB
// Warp roles.  A warp may only read the tensor-memory lanes [32 * (warp % 4), +32),
// so the eight epilogue warps form four pairs that share a lane quadrant and split
// the 32-column chunks of a tile between them (even / odd).
constexpr int kWarpLoadA = 0;
constexpr int kWarpMma = 1;
constexpr int kWarpLoadB = 2;
constexpr int kFirstEpilogueWarp = 3;
constexpr int kEpilogueWarps = 8;
constexpr int kThreads = (kFirstEpilogueWarp + kEpilogueWarps) * 32;   // 352
constexpr long long kDefaultWaitLimitCycles = 2000000000LL;   // about one second
// How the activation tile of a k-iteration is fetched.
constexpr int kModeMatrix = 0;   // rows of a plain [m, c] matrix (1x1 convolution, inner product)
constexpr int kModeIm2col = 1;   // im2col-mode tensor map: any filter, channels % 4 == 0
constexpr int kModeRows = 2;     // <= 4 channels: one filter row of 8 pixels x 4 channels per k-iteration
constexpr int kModeHalo = 3;     // stride-1 filters wider than one tap: the taps of a filter row share one pixel strip
constexpr int kModePhase = 4;    // deconvolution: one im2col convolution per phase of the output grid
constexpr int kMaxPhase = 4;      // largest deconvolution stride that phase mode takes
constexpr int kOutDirect = 0;     // how results leave: from registers,
constexpr int kOutStaged = 1;     // through shared memory as TMA tiles,
constexpr int kOutSplit = 2;      // or after a cluster's CTAs have added up their segments of the sum over K
constexpr int kOutStagedTwo = 3;  // as kOutStaged, for a launch of two layers
constexpr int kMaxHaloRows = 16; // extra strip rows ((kw - 1) * dilation) the halo mode takes

struct ConvTcArgs {
  float* out;
  int out_ld;
  int m;             // output pixels
  int cout;
  int k_iters;       // taps * c_blocks
  int c_blocks;      // ceil(c / 32)
  int kw;            // filter width (tap -> (r, s))
  int ho, wo;
  int stride_h, stride_w, pad_h, pad_w, dil_h, dil_w;
  mcb200_epilogue ep;
  // Two layers of one input in one launch: columns from second_begin on (a multiple of 32; past every column where
  // there is one layer) are the second layer's, with an output of its own.  cout counts both.
  int second_begin;
  int first_cout;    // columns of the first output
  float* second_out;
  int second_ld;
  int second_act;    // 0 none, 1 ReLU
  int* status;
  int tile_rows;     // rows of an M tile: 128 or 64, in row mode min(output width, 128)
  int row_segments;  // row mode: M tiles per output row of an image (ceil(output width / tile_rows))
  int a_bytes;       // bytes one activation tile load delivers
  int stages;        // depth of the operand ring (2 .. kMaxStages)
  int out_half;      // the output is stored as bfloat16 (else fp32), whatever the operands are
  // Halo mode.  The M index runs over a virtual output grid whose rows are `wp` = wo + (kw - 1) *
  // dil_w positions wide (the last wp - wo positions of a row are computed and never stored), so
  // that the taps s = 0 .. kw-1 of a filter row are the same strip of `128 + wp - wo` input
  // pixels read at row offsets s * dil_w.  `m` then counts virtual positions.
  int wp;
  int stage_bytes;     // activation tiles (halo mode: a strip) + weight tiles
  int stage_b_offset;  // where the weight tiles start inside a stage
  int segment_shift;   // the sum over K is made in 1, 2 or 4 segments (log2), then added up: see segment_shift_of
  int slots;           // staged epilogue: staging slots per warp, 1 or 2; 2 .. kMaxSlots when a residual is added
  int res_depth;       // and residual sub-tiles a warp requests ahead of the one it works on (1 .. slots - 1)
  int vec_store;       // the rows of output and residual can be accessed two fp32 (eight bfloat16) columns at a time
  // Grouped convolution (group_cout > 0): output columns [g * group_cout, (g + 1) * group_cout)
  // read input channels [g * group_cin, (g + 1) * group_cin).  An N tile multiplies the channels
  // its groups span (from `c_origin`, rounded down to 16 bytes) by a block-diagonal weight tile:
  // the packed weights hold zeros where an output column's group does not own the channel.
  int group_cout, group_cin;
  // Phase mode.  Output pixel (i * stride + py, j * stride + px) of a deconvolution sums the taps whose
  // row (column) has the remainder that py (px) asks for, over neighbouring input pixels: a
  // stride-1 convolution of its own per (py, px).  m runs over the (n, i, j) grid (`ho` x `wo`), an N
  // tile belongs to one phase, whose filter window starts phase_off_h[py] / phase_off_w[px] pixels
  // behind the grid's own origin.
  int phase_tiles;               // N tiles per phase
  int phase_stride_h, phase_stride_w;
  unsigned char phase_off_h[kMaxPhase], phase_off_w[kMaxPhase];
  int out_h, out_w;              // the output image, which may cut the last row and column of the grid short
  int l2_prefetch;               // ask L2 for the next tile's activations a tile ahead
  long long wait_limit;          // bound of every barrier wait, in SM cycles
  int resident_b_bytes;          // row mode: all filter rows' weight tiles stay in shared memory (bytes; 0 = streamed
                                 // with the activations).  Every M tile of such a layer multiplies the same
                                 // weights, and a third of what its ring pulled out of L2 was this one image.
  int constants_settled;         // weights and per-column constants were complete before the previous launch
                                 // began: they are fetched while that launch still runs
  int drop_last_weight_load;     // test hook: the weight producer leaves out its last k-iteration (see
                                 // mcb200_conv_test_drop_weight_load): the waits on that stage run out
};

// Optional cycle-counter trace (build with -DMCB200_CONV_TRACE): the single-thread roles and the
// first epilogue warp of CTA 0 stamp clock64() at fixed points of their loops into a device
// array that mcb200_conv_trace_read copies out.  Role 0: activation producer (per k-iteration:
// stage free, loads issued); 1: weight producer (same); 2: MMA issuer (per k-iteration: stage
// full, MMAs issued and committed); 3: epilogue warp 0 (per tile: accumulator ready, tile stored);
// 4: the same warp inside its chunk loop, five stamps per chunk (chunk begins, accumulator in registers, then staged:
// slot free / residual there, tail computed and written to the slot, store issued; from registers: tail computed, next
// residual asked for, stores issued).  A reader's buffer holds these five rows and no more.
#ifdef MCB200_CONV_TRACE
constexpr int kTraceSlots = 2048;
constexpr int kTraceRoles = 5;
__device__ long long g_conv_trace[kTraceRoles * kTraceSlots];
#define MCB200_TRACE_DECL int trace_n = 0
#define MCB200_TRACE(role)                                                                         \
  do {                                                                                             \
    if (blockIdx.x == 0 && trace_n < kTraceSlots) g_conv_trace[(role) * kTraceSlots + trace_n++] = clock64(); \
  } while (0)
#define MCB200_TRACE_CHUNK_DECL int trace_c = 0
#define MCB200_TRACE_CHUNK()                                                                       \
  do {                                                                                             \
    if (blockIdx.x == 0 && ew == 0 && lane == 0 && trace_c < kTraceSlots)                          \
      g_conv_trace[4 * kTraceSlots + trace_c++] = clock64();                                       \
  } while (0)
#else
#define MCB200_TRACE_DECL
#define MCB200_TRACE(role)
#define MCB200_TRACE_CHUNK_DECL
#define MCB200_TRACE_CHUNK()
#endif

constexpr int kMaxStages = 10;
constexpr int kMaxSlots = 4;     // every barrier here is static shared memory that the operand ring cannot use
constexpr int kSharedLimit = 232448;   // 227 KiB: the most one CTA can have on sm_100

// Shared memory of one persistent CTA is the operand ring, `stages` x (A tiles + B tiles): the copies in
// flight are what hides the round trip of a stage (L2 -> shared memory, barrier hop, MMA completion,
// barrier hop: about a microsecond).
template <int BN, int kMode, bool kPair>
struct SmemPlan {
  static constexpr int kTileBRows = kPair ? BN / 2 : BN;   // a CTA of a pair holds half of the weight tile
  static constexpr int kTileBBytes = kTileBRows * kBlockK * 4;
  // K = 32 sub-tiles per stage.  Every stage costs each single-thread role a
  // barrier wait and a signal (a few hundred cycles of pure latency), so where
  // a K = 32 step is short (narrow tiles) a stage carries two of them.
  // (Row mode keeps single steps: two filter rows per stage were measured and change nothing, its
  // tiles are bound by their epilogue.  64-column tiles as CTA pairs were measured too: slower.)
  // Halo mode: a stage is one pixel strip plus the weight tiles of a whole filter row (sized at run time).
  static constexpr int kSub =
      (kMode != kModeRows && kMode != kModeHalo && kTileABytes + kTileBBytes <= 24 * 1024) ? 2 : 1;
};

// Compile-time tag, for the activation of the fused tail (0 none, 1 ReLU, 2 per-column negative slope) and
// whether a residual is added.
template <int kValue>
struct Tag {
  static constexpr int value = kValue;
};

// Ring position of a k-iteration: stage index and the parity of its use.
// Advancing it costs an increment and a compare; the single-thread loops
// below are latency-bound on exactly this kind of scalar work.
struct RingPos {
  int stage = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void advance(int stages) {
    if (++stage == stages) {
      stage = 0;
      parity ^= 1u;
    }
  }
};

// Persistent kernel: CTA b works on tiles b, b + gridDim.x, ... (n fastest, so
// the CTAs running at one time share activation tiles through L2).  Two
// accumulators in tensor memory let the tensor core start the next tile while
// the epilogue warps drain the previous one; the TMA producers run ahead across
// tile boundaries.
//
// kPair: the CTAs of a cluster of two share one tcgen05.mma.cta_group::2 per
// K=8 step.  The pair works on 256 output pixels (128 per CTA) x BN channels;
// each CTA fetches its own activation tile and only half of the weight tile, the
// rank-0 CTA issues the MMAs for both, and each CTA drains its own half of the
// result from its own tensor memory.  Weight bytes per MAC halve, which is what
// bounds the layers whose operands come out of L2 faster than the ring can
// turn over.  Barriers that both CTAs signal (stage full, accumulator drained)
// live in rank 0; tcgen05.commit delivers the arrivals that both CTAs wait on to
// each CTA's own copy of the barrier.
//
// kHalf: activations, weights and the residual are bfloat16 (tcgen05.mma
// kind::f16, fp32 accumulation); a k-iteration then covers 64 channels in the
// same 128-byte rows.  Independently of that, the output is stored as fp32 or
// as bfloat16 (args.out_half).
template <int BN, int kMode, bool kPair, bool kHalf, int kOut>
__global__ void __launch_bounds__(kThreads, 1)
conv_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_out, const __grid_constant__ CUtensorMap map_res,
               const ConvTcArgs args) {
  constexpr bool kStaged = kOut == kOutStaged || kOut == kOutStagedTwo, kSplit = kOut == kOutSplit;
  // Layers whose sum over K is cut into segments (segment_shift_of): these modes.
  constexpr bool kSegments = !kStaged && (kMode == kModeMatrix || kMode == kModeIm2col || kMode == kModeHalo);
  // May hold two layers.  (The staged form is compiled for either: asked per chunk whose columns it has, it was 4 to 9 % slower
  // for every launch of one layer that its epilogue bounds, bfloat16 above all: 64 -> 128 at 56 x 56, batch 64 21.9 us, 19.9 so.)
  constexpr bool kTwo = (kMode == kModeMatrix || kMode == kModeIm2col || kMode == kModeHalo) && kOut != kOutStaged;
  static_assert(!kSplit || (kSegments && !kPair), "a split tile belongs to one CTA per segment");
  static_assert(!(kStaged && (BN < 64 || kMode == kModeHalo || kMode == kModePhase)), "a staged tile is one box of the output");
  static_assert(!(kPair && kMode == kModeRows), "row mode runs unpaired");
  static_assert(!(kHalf && kMode == kModeRows), "row mode takes fp32 images");
  static_assert(!((kPair || kHalf) && kMode == kModePhase), "phase mode runs unpaired on fp32 operands");
  constexpr bool kIm2col = kMode == kModeIm2col || kMode == kModePhase;     // how activations are fetched
  constexpr bool kScatter = kMode == kModeHalo || kMode == kModePhase;      // output rows are not one box
  using Plan = SmemPlan<BN, kMode, kPair>;
  constexpr int kElemsK = kHalf ? kBlockKHalf : kBlockK;   // channels per k-iteration
  const int stages = args.stages;
  const long long wait_limit = args.wait_limit;   // SM cycles a barrier wait may take before the CTA gives up

  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[kMaxStages];    // both operand tiles of a stage have landed (two producers)
  __shared__ uint64_t empty_bar[kMaxStages];   // the MMAs reading a stage have retired
  __shared__ uint64_t tmem_full_bar[2];
  __shared__ uint64_t tmem_empty_bar[2];
  __shared__ uint64_t res_bar[kStaged ? kEpilogueWarps : 1][kMaxSlots];   // per epilogue warp, per staging slot
  __shared__ uint64_t col_bar[2];              // per-column table of a tile is complete
  __shared__ uint64_t wres_bar;                // row mode: the resident weight tiles have landed
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ __align__(16) float col_scale[2][BN];   // per-column constants of the current tiles
  __shared__ __align__(16) float col_shift[2][BN];
  __shared__ __align__(16) float col_slope[2][BN];

  // 128-byte swizzled tiles must start on a 1024-byte boundary.
  const uint32_t raw_addr = smem_addr(smem_raw);
  uint8_t* tiles = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  constexpr bool kOrdinary = kStaged && kMode != kModeRows;   // tiles of 128 rows, nothing resident: a stage of fixed size
  const int stage_bytes = kOrdinary ? Plan::kSub * (kTileABytes + Plan::kTileBBytes) : args.stage_bytes;
  const int stage_b_offset = kOrdinary ? Plan::kSub * kTileABytes : args.stage_b_offset;
  const int a_sub_bytes = stage_b_offset / Plan::kSub;   // sub-tiles of a stage: [A ...][B ...]
  const bool resident_b = kMode == kModeRows && args.resident_b_bytes > 0;
  uint8_t* resident = tiles + stages * stage_bytes;   // stages are multiples of 1024 bytes: so is this address
  uint8_t* staging_base = resident + (kMode == kModeRows ? args.resident_b_bytes : 0);
  uint8_t* exchange = staging_base;                   // split form: the cluster's partial sums of what this CTA finishes

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_tiles = kMode == kModePhase ? args.phase_tiles * args.phase_stride_h * args.phase_stride_w
                                          : (args.cout + BN - 1) / BN;
  // Rows of an M tile: with 64, tcgen05.mma runs at M = 64 and its accumulator lies in the first 16 lanes of
  // each tensor-memory quadrant (row 16 * quadrant + lane).
  constexpr bool kShortTiles = !kPair && !kStaged && (kMode == kModeMatrix || kMode == kModeIm2col || kMode == kModeHalo);
  const int tile_m = kShortTiles ? args.tile_rows : kBlockM;
  const int warp_rows = kShortTiles ? args.tile_rows >> 2 : 32;   // rows an epilogue warp owns: one quadrant's
  // Row mode: an M tile is (a segment of at most 128 pixels of) one output row of one image.
  const int m_tiles = kMode == kModeRows ? (args.m / args.wo) * args.row_segments : (args.m + tile_m - 1) / tile_m;
  // Row mode helpers: image row (n * ho + p) and first pixel of the segment of M tile mt.
  auto row_of = [&](int mt) { return mt / args.row_segments; };
  auto seg_start = [&](int mt) { return (mt % args.row_segments) * args.tile_rows; };
  // A work unit is an M tile (or a pair of neighbouring M tiles) x an N tile;
  // `worker` is the CTA (or pair) index among `workers`.
  const uint32_t rank = kPair ? cluster_cta_rank() : 0u;
  // A cluster of 2 or 4 CTAs splits a tile's sum over K, a segment each.
  const uint32_t split_rank = kSplit ? cluster_cta_rank() : 0u;
  const int cluster_shift = kPair ? 1 : kSplit ? args.segment_shift : 0;
  const int worker = static_cast<int>(blockIdx.x) >> cluster_shift;
  const int workers = static_cast<int>(gridDim.x) >> cluster_shift;
  // This CTA's k-iterations, and the first of segment i.
  const int segments = kSegments ? 1 << args.segment_shift : 1;
  auto segment_begin = [&](int i) { return kSegments ? (args.k_iters * i) >> args.segment_shift : i * args.k_iters; };
  const int first_segment = kSplit ? static_cast<int>(split_rank) : 0;
  const int k_begin = segment_begin(first_segment), k_end = kSplit ? segment_begin(first_segment + 1) : args.k_iters;
  // Tensor memory: an accumulator per segment, twice where that fits (one is then drained while the other fills).
  const int accumulators = kSegments && !kSplit && segments * BN > 256 ? 1 : 2;
  const int acc_columns = kSplit ? BN : segments * BN;
  const int m_units = kPair ? (m_tiles + 1) >> 1 : m_tiles;
  const int num_tiles = n_tiles * m_units;
  auto unit_to_mt = [&](int unit) { return kPair ? 2 * unit + static_cast<int>(rank) : unit; };

  // Some twenty barriers: a thread each (one thread doing them all costs every launch most of a
  // microsecond before its first load can go out).
  {
    const int t = static_cast<int>(threadIdx.x);
    if (t == 0) abort_flag = 0;
    if (t < stages) {
      mbar_init(&full_bar[t], resident_b ? 1 : 2);     // one arrival per producer thread that fills the stage
      mbar_init(&empty_bar[t], 1);
      fence_barrier_init();
    } else if (t >= 32 && t < 34) {
      const int b = t - 32;
      mbar_init(&tmem_full_bar[b], 1);
      mbar_init(&tmem_empty_bar[b], kPair ? 2 * kEpilogueWarps : kEpilogueWarps);   // one arrival per epilogue warp
      mbar_init(&col_bar[b], kEpilogueWarps);
      fence_barrier_init();
    } else if (kStaged && t >= 64 && t < 64 + kEpilogueWarps * kMaxSlots) {
      mbar_init(&res_bar[(t - 64) / kMaxSlots][(t - 64) % kMaxSlots], 1);
      fence_barrier_init();
    } else if (t == 34) {
      tma_prefetch_descriptor(&map_a);
      tma_prefetch_descriptor(&map_b);
    } else if (t == 35) {
      mbar_init(&wres_bar, 1);
      fence_barrier_init();
    }
  }
  if (warp == kWarpMma) {
    tmem_alloc(&tmem_base_slot, static_cast<uint32_t>(accumulators * acc_columns));
    tmem_relinquish();
  }
  tc_fence_before_sync();
  if (kPair || kSplit) {
    cluster_sync_all();   // the peers run, and their barriers are initialised before anything signals them
  } else {
    __syncthreads();
  }
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  volatile int* abort = &abort_flag;
  // A paired MMA writes the same tensor-memory address in both CTAs.  Each CTA
  // makes the first and only allocation of its SM, which starts at column 0;
  // anything else is refused rather than computed wrongly.
  // Up to here the CTA has only set itself up, which may overlap the tail of
  // the previous launch of the stream; from here on it touches tensors.  What the previous launch
  // cannot have written, the weights and the per-column constants of a layer that has run before, need
  // not wait for its end: the weight producer fills the ring and the epilogue warps their first table
  // while the activations are still being computed.  (At batch 1 a layer is a few microseconds of
  // latency, one of which was the weights' first trip out of DRAM and 0.4 the table's.)
  grid_launch_dependents();
  const bool early = args.constants_settled != 0;
  if (!early || (warp != kWarpLoadB && warp < kFirstEpilogueWarp)) grid_dependency_wait();
  const bool usable = !kPair || tmem_base == 0u;
  if (!usable && threadIdx.x == 0) abort_flag = 1;
  // Cluster-window addresses of rank 0's shared barriers.
  const uint32_t full_bar_leader = kPair ? cluster_map(smem_addr(&full_bar[0]), 0u) : 0u;
  const uint32_t tmem_empty_leader = kPair ? cluster_map(smem_addr(&tmem_empty_bar[0]), 0u) : 0u;

  // After an abort: give a producer's copies that are still in flight a bounded
  // time to land before the CTA's shared memory is released.
  auto drain_loads = [&](int issued) {
    if (!*abort) return;
    const int first = issued > stages ? issued - stages : 0;
    for (int j = first; j < issued; ++j) {
      const long long start = clock64();
      while (!mbar_try_wait(&full_bar[j % stages], static_cast<uint32_t>(j / stages) & 1u)) {
        if (clock64() - start > wait_limit / 8) break;
      }
    }
  };

  if (!usable) {
    // fall through to the teardown; the peer's waits run out and it follows
  } else if (warp == kWarpLoadA) {
    // ------------------------------------------------------------ activation tiles
    if (elect_one()) {
      RingPos pos;
      int issued = 0;
      bool alive = true;
      MCB200_TRACE_DECL;
      const uint32_t a_bytes = static_cast<uint32_t>(args.a_bytes);
      for (int tile = worker; tile < num_tiles && alive; tile += workers) {
        const int mt = unit_to_mt(tile / n_tiles);
        const int m0 = mt * tile_m;
        // The odd M tile out at the end of a paired launch has no pixels: its
        // CTA loads nothing, and the MMA computes rows nobody stores.
        const bool live = !kPair || mt < m_tiles;
        // Only rank 0's barrier counts bytes: its producers announce what both
        // CTAs are about to fetch, the peer's copies just report completion
        // there (a remote arrival per k-iteration would cost the peer's
        // producer a cluster-scope release, about a microsecond each).
        const uint32_t announce =
            !kPair ? a_bytes : (rank != 0u ? 0u : (mt + 1 < m_tiles ? 2u * a_bytes : a_bytes));
        int base_w = 0, base_h = 0, base_n = 0;
        if (kMode == kModeRows) {
          const int row = row_of(mt);
          base_n = row / args.ho;
          base_h = (row - base_n * args.ho) * args.stride_h;   // row in the spatially padded copy
          base_w = seg_start(mt);                              // first output pixel of the segment
        }
        if (kIm2col) {
          const int q = m0 % args.wo;
          const int p = (m0 / args.wo) % args.ho;
          base_n = m0 / (args.wo * args.ho);
          base_w = q * args.stride_w - args.pad_w;
          base_h = p * args.stride_h - args.pad_h;
        }
        if (kMode == kModeHalo) {
          // m0 is a position of the virtual output grid (rows of wp positions, stride 1)
          const int t = m0 / args.wp;
          base_n = t / args.ho;
          base_w = m0 - t * args.wp - args.pad_w;
          base_h = t - base_n * args.ho - args.pad_h;
        }
        // First channel the tile's weight columns refer to (grouped layers: the first channel of
        // the first group the N tile touches, rounded down to a 16-byte boundary of the pixel).
        int c_origin = 0;
        if (args.group_cout > 0) {
          const int n0 = (tile % n_tiles) * BN;
          c_origin = ((n0 / args.group_cout) * args.group_cin) & ~((kHalf ? 8 : 4) - 1);
        }
        // The activations of this CTA's next tile are asked for now, a tile ahead (L2 prefetch, no
        // shared memory, nothing to wait for).  A tile always brings pixels nobody has read yet,
        // the ring looks only a few stages ahead, and a load that waits for DRAM holds up the whole
        // in-order ring behind it.  Of the CTAs that share an M tile (one per N tile) the one
        // with N tile 0 asks; grouped layers read other channels per N tile, so there every CTA asks.
        if (args.l2_prefetch && kMode != kModeRows) {
          const int next = tile + workers;
          const int n_index = next % n_tiles;
          const int mt2 = next < num_tiles ? unit_to_mt(next / n_tiles) : m_tiles;
          if (mt2 < m_tiles && (n_index == 0 || args.group_cout > 0)) {
            const int origin2 = args.group_cout > 0
                                    ? (((n_index * BN) / args.group_cout) * args.group_cin) & ~((kHalf ? 8 : 4) - 1)
                                    : 0;
            const int v2 = mt2 * tile_m;
            if (kMode == kModeMatrix) {
              for (int cb = 0; cb < args.c_blocks; ++cb) tma_prefetch_2d(&map_a, origin2 + cb * kElemsK, v2);
            } else {
              int w2, h2, n2;
              if (kMode == kModeHalo) {
                const int t2 = v2 / args.wp;
                n2 = t2 / args.ho;
                w2 = v2 - t2 * args.wp - args.pad_w;
                h2 = t2 - n2 * args.ho - args.pad_h;
              } else {
                n2 = v2 / (args.wo * args.ho);
                w2 = (v2 % args.wo) * args.stride_w - args.pad_w;
                h2 = ((v2 / args.wo) % args.ho) * args.stride_h - args.pad_h;
              }
              const int kh = kMode == kModeHalo ? args.k_iters / args.c_blocks : args.k_iters / (args.c_blocks * args.kw);
              // im2col mode: the middle tap column of every filter row touches (nearly) every pixel
              // the other columns touch; with a stride, its neighbour column takes the pixels between.
              const int s_mid = kMode == kModeHalo ? 0 : args.kw / 2;
              const int s_count = (kMode == kModeIm2col && args.stride_w > 1 && args.kw > 1) ? 2 : 1;
              for (int r = 0; r < kh; ++r)
                for (int sc = 0; sc < s_count; ++sc)
                  for (int cb = 0; cb < args.c_blocks; ++cb)
                    tma_prefetch_im2col_4d(&map_a, origin2 + cb * kElemsK, w2, h2, n2,
                                           static_cast<uint16_t>(min(s_mid + sc, args.kw - 1) * args.dil_w),
                                           static_cast<uint16_t>(r * args.dil_h));
            }
          }
        }
        // Position inside the filter, advanced incrementally: channel block,
        // then tap column, then tap row.
        int c0 = 0, sx = 0;
        uint16_t off_w0 = 0, off_h = 0;
        if (kMode == kModePhase) {
          const int phase = (tile % n_tiles) / args.phase_tiles;
          const int py = phase / args.phase_stride_w;
          off_h = args.phase_off_h[py];
          off_w0 = args.phase_off_w[phase - py * args.phase_stride_w];
        }
        uint16_t off_w = off_w0;
        int row_h = base_h;
        if (kSplit && k_begin > 0) {   // the segment's first position inside the filter
          const int tap = k_begin / args.c_blocks;
          c0 = (k_begin - tap * args.c_blocks) * kElemsK;
          if (kMode == kModeHalo) off_h = static_cast<uint16_t>(tap * args.dil_h);
          if (kMode == kModeIm2col) {
            off_h = static_cast<uint16_t>(tap / args.kw * args.dil_h);
            sx = tap % args.kw;
            off_w = static_cast<uint16_t>(sx * args.dil_w);
          }
        }
        int segment = first_segment, segment_end = segment_begin(first_segment + 1), nsub = 0;
        for (int k = k_begin; k < k_end; k += nsub) {
          if (!mbar_wait_bounded(&empty_bar[pos.stage], pos.parity ^ 1u, abort, wait_limit)) {
            alive = false;
            break;
          }
          MCB200_TRACE(0);
          nsub = Plan::kSub == 1 ? 1 : min(segment_end - k, Plan::kSub);   // (a constant step keeps the loop short)
          if (kSegments && k + nsub == segment_end) segment_end = segment_begin(++segment + 1);
          uint8_t* a_dst = tiles + pos.stage * stage_bytes;
          uint64_t* bar = &full_bar[pos.stage];
          const uint32_t bar_leader = full_bar_leader + static_cast<uint32_t>(pos.stage) * 8u;
          if (rank == 0u) mbar_expect_tx(bar, announce * static_cast<uint32_t>(nsub));
#pragma unroll
          for (int j = 0; j < Plan::kSub; ++j) {
            if (j >= nsub) break;
            if (kMode == kModeRows) {
              // A sub-tile is one filter row: tile_rows pixels x (8 pixels x 4 channels) of a padded input row.
              tma_load_4d(&map_a, bar, a_dst, 0, base_w, row_h, base_n);   // pixels past the row read as zero
              row_h += args.dil_h;
            } else if (kMode == kModeHalo) {
              // One strip of 128 + halo pixels x one channel block, at filter row off_h: every tap
              // of that row reads it (k-iterations run over filter rows x channel blocks).
              if (kPair) {
                if (live) tma_load_im2col_4d_pair(&map_a, bar_leader, a_dst, c_origin + c0, base_w, base_h, base_n, 0, off_h);
              } else {
                tma_load_im2col_4d(&map_a, bar, a_dst, c_origin + c0, base_w, base_h, base_n, 0, off_h);
              }
              c0 += kElemsK;
              if (c0 >= args.c_blocks * kElemsK) {
                c0 = 0;
                off_h = static_cast<uint16_t>(off_h + args.dil_h);
              }
            } else if (kIm2col) {
              if (kPair) {
                if (live) tma_load_im2col_4d_pair(&map_a, bar_leader, a_dst, c_origin + c0, base_w, base_h, base_n, off_w, off_h);
              } else {
                tma_load_im2col_4d(&map_a, bar, a_dst, c_origin + c0, base_w, base_h, base_n, off_w, off_h);
              }
              c0 += kElemsK;
              if (c0 >= args.c_blocks * kElemsK) {
                c0 = 0;
                off_w = static_cast<uint16_t>(off_w + args.dil_w);
                if (++sx == args.kw) {
                  sx = 0;
                  off_w = off_w0;
                  off_h = static_cast<uint16_t>(off_h + args.dil_h);
                }
              }
            } else {
              if (kPair) {
                if (live) tma_load_2d_pair(&map_a, bar_leader, a_dst, c_origin + c0, m0);
              } else {
                tma_load_2d(&map_a, bar, a_dst, c_origin + c0, m0);
              }
              c0 += kElemsK;
            }
            a_dst += a_sub_bytes;
          }
          MCB200_TRACE(0);
          ++issued;
          pos.advance(stages);
        }
      }
      drain_loads(issued);
    }
  } else if (warp == kWarpLoadB) {
    // ------------------------------------------------------------ weight tiles
    if (elect_one()) {
      RingPos pos;
      int issued = 0;
      bool alive = true;
      MCB200_TRACE_DECL;
      if (resident_b) {
        // All filter rows at once, into their own region; the ring then carries activations only.
        const int loads = args.drop_last_weight_load ? args.k_iters - 1 : args.k_iters;
        mbar_expect_tx(&wres_bar, Plan::kTileBBytes * static_cast<uint32_t>(args.k_iters));
        for (int k = 0; k < loads; ++k) tma_load_2d(&map_b, &wres_bar, resident + k * Plan::kTileBBytes, k * kElemsK, 0);
        // The copies land before this CTA may release its shared memory (bounded, like every wait).
        const long long start = clock64();
        while (!mbar_try_wait(&wres_bar, 0u)) {
          if (clock64() - start > wait_limit) break;
        }
        alive = false;   // nothing to stream
      }
      for (int tile = worker; tile < num_tiles && alive; tile += workers) {
        // A CTA of a pair fetches the half of the weight tile that matches its rank.
        int n0 = (tile % n_tiles) * BN + static_cast<int>(rank) * Plan::kTileBRows;
        if (kMode == kModePhase) {
          // weight rows run over the phases, then their output channels
          const int phase = (tile % n_tiles) / args.phase_tiles;
          n0 = phase * args.cout + (tile % n_tiles - phase * args.phase_tiles) * BN;
        }
        int k0 = 0;
        int halo_cb = 0, halo_row_k0 = 0;   // halo mode: channel block and first packed-weight column of the filter row
        if (kSplit && kMode == kModeHalo) {
          const int row = k_begin / args.c_blocks;
          halo_cb = k_begin - row * args.c_blocks;
          halo_row_k0 = row * args.kw * args.c_blocks * kElemsK;
        } else if (kSplit) {
          k0 = k_begin * kElemsK;
        }
        int segment = first_segment, segment_end = segment_begin(first_segment + 1), nsub = 0;
        for (int k = k_begin; k < k_end; k += nsub) {
          if (!mbar_wait_bounded(&empty_bar[pos.stage], pos.parity ^ 1u, abort, wait_limit)) {
            alive = false;
            break;
          }
          MCB200_TRACE(1);
          nsub = Plan::kSub == 1 ? 1 : min(segment_end - k, Plan::kSub);   // (a constant step keeps the loop short)
          if (kSegments && k + nsub == segment_end) segment_end = segment_begin(++segment + 1);
          if (args.drop_last_weight_load && tile + workers >= num_tiles && k + nsub >= k_end) {
            alive = false;   // nothing arrives on this stage's barrier: every role's wait on it is bounded
            break;
          }
          uint8_t* b_dst = tiles + pos.stage * stage_bytes + stage_b_offset;
          uint64_t* bar = &full_bar[pos.stage];
          const uint32_t bar_leader = full_bar_leader + static_cast<uint32_t>(pos.stage) * 8u;
          if (kMode == kModeHalo) {
            // The weight tiles of the kw taps of this filter row for this channel block.  Packed
            // weight columns run [tap][channel block]; tap = row * kw + s.
            const int row_stride = args.c_blocks * kElemsK;
            if (rank == 0u) mbar_expect_tx(bar, (kPair ? 2u : 1u) * Plan::kTileBBytes * static_cast<uint32_t>(args.kw));
            int kcol = halo_row_k0 + halo_cb * kElemsK;
            for (int s = 0; s < args.kw; ++s) {
              if (kPair) {
                tma_load_2d_pair(&map_b, bar_leader, b_dst, kcol, n0);
              } else {
                tma_load_2d(&map_b, bar, b_dst, kcol, n0);
              }
              kcol += row_stride;
              b_dst += Plan::kTileBBytes;
            }
            if (++halo_cb == args.c_blocks) {
              halo_cb = 0;
              halo_row_k0 += args.kw * row_stride;
            }
            MCB200_TRACE(1);
            ++issued;
            pos.advance(stages);
            continue;
          }
          // Rank 0 announces both halves of a paired weight tile.
          if (rank == 0u) mbar_expect_tx(bar, (kPair ? 2u : 1u) * Plan::kTileBBytes * static_cast<uint32_t>(nsub));
#pragma unroll
          for (int j = 0; j < Plan::kSub; ++j) {
            if (j >= nsub) break;
            if (kPair) {
              tma_load_2d_pair(&map_b, bar_leader, b_dst, k0, n0);
            } else {
              tma_load_2d(&map_b, bar, b_dst, k0, n0);
            }
            k0 += kElemsK;
            b_dst += Plan::kTileBBytes;
          }
          MCB200_TRACE(1);
          ++issued;
          pos.advance(stages);
        }
      }
      drain_loads(issued);
    }
  } else if (warp == kWarpMma) {
    // ------------------------------------------------------------ MMA issuer
    if ((!kPair || rank == 0u) && elect_one()) {
      constexpr uint32_t idesc_full = kHalf ? umma_idesc_bf16(kPair ? 2 * kBlockM : kBlockM, BN)
                                            : umma_idesc_tf32(kPair ? 2 * kBlockM : kBlockM, BN);
      constexpr uint32_t idesc_small = kHalf ? umma_idesc_bf16(kSmallM, BN) : umma_idesc_tf32(kSmallM, BN);
      const uint32_t idesc = kShortTiles && tile_m == kSmallM ? idesc_small : idesc_full;
      RingPos pos;
      int local = 0;   // tiles done by this CTA
      bool alive = true;
      MCB200_TRACE_DECL;
      const uint32_t tiles_addr = smem_addr(tiles);
      if (resident_b) {
        if (!mbar_wait_bounded(&wres_bar, 0u, abort, wait_limit)) alive = false;
        tc_fence_after_sync();
      }
      for (int tile = worker; tile < num_tiles && alive; tile += workers, ++local) {
        const int ab = accumulators == 2 ? local & 1 : 0;
        const uint32_t use = static_cast<uint32_t>(accumulators == 2 ? local >> 1 : local) & 1u;
        // The epilogue must have drained this accumulator (first use passes).
        if (!mbar_wait_bounded(&tmem_empty_bar[ab], use ^ 1u, abort, wait_limit)) break;
        tc_fence_after_sync();
        uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(ab * acc_columns);
        uint32_t accumulate = 0;
        int segment = first_segment, segment_end = segment_begin(first_segment + 1), nsub = 0;
        for (int k = k_begin; k < k_end; k += nsub) {
          if (!mbar_wait_bounded(&full_bar[pos.stage], pos.parity, abort, wait_limit)) {
            alive = false;
            break;
          }
          tc_fence_after_sync();
          MCB200_TRACE(2);
          nsub = Plan::kSub == 1 ? 1 : min(segment_end - k, Plan::kSub);   // (a constant step keeps the loop short)
          const uint32_t a_addr = tiles_addr + static_cast<uint32_t>(pos.stage * stage_bytes);
          uint64_t desc_a = umma_desc_k_sw128(a_addr);
          uint64_t desc_b = umma_desc_k_sw128(
              resident_b ? smem_addr(resident) + static_cast<uint32_t>(k) * Plan::kTileBBytes : a_addr + stage_b_offset);
          if (kMode == kModeHalo) {
            // Tap s of the filter row reads the strip s * dil_w pixel rows (128 bytes each) further
            // down: the same swizzled bytes, another start address.  The swizzle is a function of
            // the shared-memory address itself (TMA wrote the strip that way and the tensor core
            // reads it that way), so a start address that is not a multiple of the 1024-byte
            // pattern needs nothing else: the descriptor's base-offset field stays 0 (measured:
            // results equal the im2col mode's; with (address >> 7) & 7 in that field they are wrong).
            const uint32_t tap_step = static_cast<uint32_t>(args.dil_w) * 128u;
            for (int s = 0; s < args.kw; ++s) {
              const uint64_t da = umma_desc_k_sw128(a_addr + static_cast<uint32_t>(s) * tap_step);
#pragma unroll
              for (int kk = 0; kk < kMmaPerBlock; ++kk) {
                if (kHalf) {
                  if (kPair) {
                    umma_bf16_pair(tmem_acc, da + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
                  } else {
                    umma_bf16(tmem_acc, da + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
                  }
                } else if (kPair) {
                  umma_tf32_pair(tmem_acc, da + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
                } else {
                  umma_tf32(tmem_acc, da + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
                }
                accumulate = 1u;
              }
              desc_b += Plan::kTileBBytes >> 4;
            }
          }
#pragma unroll
          for (int j = 0; j < Plan::kSub; ++j) {
            if (kMode == kModeHalo) break;
            if (j >= nsub) break;
#pragma unroll
            for (int kk = 0; kk < kMmaPerBlock; ++kk) {
              // Each K step (8 tf32 or 16 bf16) is 32 bytes further along the swizzled
              // row: +2 in the descriptor's 16-byte address units.
              if (kHalf) {
                if (kPair) {
                  umma_bf16_pair(tmem_acc, desc_a + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
                } else {
                  umma_bf16(tmem_acc, desc_a + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
                }
              } else if (kPair) {
                umma_tf32_pair(tmem_acc, desc_a + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
              } else {
                umma_tf32(tmem_acc, desc_a + 2 * kk, desc_b + 2 * kk, idesc, accumulate);
              }
              accumulate = 1u;
            }
            desc_a += a_sub_bytes >> 4;            // next sub-tile (start address is in 16-byte units)
            desc_b += Plan::kTileBBytes >> 4;
          }
          if (kPair) {
            umma_commit_pair(&empty_bar[pos.stage], 3);   // both CTAs' producers wait on their own copy
          } else {
            umma_commit(&empty_bar[pos.stage]);
          }
          MCB200_TRACE(2);
          if (kSegments && k + nsub == segment_end) {   // the next segment sums in an accumulator of its own
            segment_end = segment_begin(++segment + 1);
            tmem_acc += BN;
            accumulate = 0;
          }
          pos.advance(stages);
        }
        if (alive) {
          if (kPair) {
            umma_commit_pair(&tmem_full_bar[ab], 3);
          } else {
            umma_commit(&tmem_full_bar[ab]);
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int ew = warp - kFirstEpilogueWarp;   // 0..7
    const int quad = warp & 3;                  // tensor-memory lanes [32*quad, 32*quad+32)
    const int half = ew >> 2;                   // chunks half, half + 2, ... of every tile
    const mcb200_epilogue& ep = args.ep;
    const bool has_res = ep.residual != nullptr;
    constexpr int kChunk = BN >= 64 ? 32 : 16;  // columns of a chunk: both warps of a quadrant have one
    constexpr int kChunks = BN / kChunk;
    constexpr int kGroups = kChunk / 8;         // a chunk comes out of tensor memory in groups of eight columns
    // Of group j a lane holds columns 8 j + col_in and the next, of rows row_in + 8 i (i < row_sets).
    const int col_in = 2 * (lane & 3);
    const int row_in = lane >> 2;
    const int row_sets = kShortTiles ? warp_rows >> 3 : 4;
    const bool vec = args.vec_store != 0;
    const int epi_tid = threadIdx.x - kFirstEpilogueWarp * 32;   // 0..255 over the epilogue warps
    // 0: no activation, 1: plain ReLU, 2: per-column negative slope (leaky ReLU / PReLU)
    const int act_mode = ep.act == 0 ? 0 : ((ep.act == 1 && ep.slope == 0.f) ? 1 : 2);

    // First column of a tile, and the output rows (-1: none) of this lane's row sets.
    auto tile_n0 = [&](int tile) {
      const int nt = tile % n_tiles;
      return (kMode == kModePhase ? nt % args.phase_tiles : nt) * BN;
    };
    auto tile_rows = [&](int tile, int (&rows)[4]) {
      const int unit = tile / n_tiles;
      const int mt = unit_to_mt(unit);
      // First output row (pixel) of this warp's slice of the tile, and how many of its rows exist.
      const int row0 = (kMode == kModeRows ? row_of(mt) * args.wo + seg_start(mt) : mt * tile_m) + quad * warp_rows;
      const int rows_here = kMode == kModeRows ? min(args.tile_rows, args.wo - seg_start(mt)) - quad * 32
                                               : min(args.m - row0, warp_rows);
      if (!kScatter) {
#pragma unroll
        for (int i = 0; i < 4; ++i) rows[i] = row_in + 8 * i < rows_here ? row0 + row_in + 8 * i : -1;
        return;
      }
      // A division or two per tile and lane: lane r works out row r and hands it to the lanes that store it.
      int mine = row0 + lane;
      bool ok = lane < rows_here;
      if (kMode == kModeHalo) {
        const int t = mine / args.wp;              // (image, output row); `mine` counts virtual positions
        const int j = mine - t * args.wp;
        ok = ok && j < args.wo;
        mine = t * args.wo + j;
      }
      if (kMode == kModePhase) {
        const int phase = (tile - unit * n_tiles) / args.phase_tiles;
        const int phase_y = phase / args.phase_stride_w;
        const int t = mine / args.wo;              // (image, grid row)
        const int image = t / args.ho;
        const int y = (t - image * args.ho) * args.phase_stride_h + phase_y;
        const int x = (mine - t * args.wo) * args.phase_stride_w + (phase - phase_y * args.phase_stride_w);
        ok = ok && y < args.out_h && x < args.out_w;
        mine = (image * args.out_h + y) * args.out_w + x;
      }
      if (!ok) mine = -1;
#pragma unroll
      for (int i = 0; i < 4; ++i) rows[i] = __shfl_sync(0xffffffffu, mine, (row_in + 8 * i) & 31);
    };
    // The residual of the chunk at col0, asked for a chunk ahead: a DRAM round trip (one to two microseconds)
    // that the chunk before it, or the main loop of a first chunk, hides.
    float res[4][kGroups][2];
    auto fetch_residual = [&](const int (&rows)[4], int col0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i >= row_sets) break;
        const size_t at = static_cast<size_t>(rows[i] < 0 ? 0 : rows[i]) * ep.residual_ld + col0 + col_in;
#pragma unroll
        for (int j = 0; j < kGroups; ++j) {
          const int c = col0 + 8 * j + col_in;
          float2 r = make_float2(0.f, 0.f);
          if (rows[i] >= 0 && c < args.cout) {
            if (kHalf) {
              const uint16_t* src = reinterpret_cast<const uint16_t*>(ep.residual) + at + 8 * j;
              if (vec) {
                const uint32_t w = *reinterpret_cast<const uint32_t*>(src);
                r = make_float2(bf16_lo(w), bf16_hi(w));
              } else {
                r.x = bf16_lo(src[0]);
                if (c + 1 < args.cout) r.y = bf16_lo(src[1]);
              }
            } else {
              const float* src = ep.residual + at + 8 * j;
              if (vec) {
                r = *reinterpret_cast<const float2*>(src);
              } else {
                r.x = src[0];
                if (c + 1 < args.cout) r.y = src[1];
              }
            }
          }
          res[i][j][0] = r.x;
          res[i][j][1] = r.y;
        }
      }
    };
    int table_n0[2] = {-1, -1};          // first column the per-column tables were filled for
    uint32_t table_fills[2] = {0u, 0u};
    auto fill_table = [&](int ab, int n0) {
      for (int c = epi_tid; c < BN; c += kEpilogueWarps * 32) {
        const int cc = n0 + c;
        const bool in = cc < args.cout;
        col_scale[ab][c] = (in && ep.scale) ? __ldg(ep.scale + cc) : 1.f;
        col_shift[ab][c] = (in && ep.shift) ? __ldg(ep.shift + cc) : 0.f;
        col_slope[ab][c] = ep.act == 2 ? ((in && ep.prelu) ? __ldg(ep.prelu + (ep.prelu_shared ? 0 : cc)) : 0.f) : ep.slope;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&col_bar[ab]);
      table_n0[ab] = n0;
    };
    // The first tile's table, before anything else is waited for.
    if (worker < num_tiles) fill_table(0, tile_n0(worker));
    if (early) grid_dependency_wait();
    int rows[4] = {-1, -1, -1, -1};
    if (!kStaged && worker < num_tiles) {
      tile_rows(worker, rows);
      if (!kSplit && has_res) fetch_residual(rows, tile_n0(worker) + half * kChunk);
    }

    // Staged form.  A slot holds a 32 x 32 sub-tile: 4 KiB, or 2 KiB when residual and result are both bfloat16.
    const int slots = args.slots;
    const int slot_bytes = (kHalf && args.out_half) ? 2048 : 4096;
    uint8_t* staging = staging_base + ew * (slots * slot_bytes);
    auto slot_ptr = [&](int slot) { return reinterpret_cast<float*>(staging + slot * slot_bytes); };
    // Chunk sequence of this warp: for each of its CTA's tiles, the 32-column
    // chunks it owns that exist (the last n-tile may have fewer), left to right.
    // `seq` numbers them.  With a residual the warp cycles through its staging
    // slots, and a cursor of lane 0 walks the same sequence a few chunks ahead of
    // the computation (args.res_depth): it copies a coming chunk's residual
    // sub-tile into the slot that comes free next.  Asking L2 for the residual
    // further ahead instead (cp.async.bulk.prefetch) was tried and removed: the
    // lines were evicted by the output stream before use and DRAM reads grew by
    // half.
    struct ChunkCursor {
      int local;   // how many of this CTA's tiles lie behind the cursor
      int chunk;   // next chunk of the current tile
      int mt;      // M tile and first column of the current tile (-1: not looked up yet)
      int n0;
    };
    auto cursor_next = [&](ChunkCursor& cur, int& mt, int& col) {
      for (;;) {
        if (cur.mt < 0) {   // entering a tile: one division per tile, none per chunk
          const int tile = worker + cur.local * workers;
          if (tile >= num_tiles) return false;
          const int unit = tile / n_tiles;
          cur.mt = unit_to_mt(unit);
          cur.n0 = (tile - unit * n_tiles) * BN;
        }
        col = cur.n0 + cur.chunk * 32;
        if (cur.chunk >= kChunks || col >= args.cout) {   // this warp's chunks of the tile are done
          cur.chunk = half;
          ++cur.local;
          cur.mt = -1;
          continue;
        }
        mt = cur.mt;
        cur.chunk += 2;
        return true;
      }
    };
    ChunkCursor ld = {0, half, -1, 0};
    int ld_slot = 0;                     // slot of the next residual load
    int cur_slot = 0;                    // slot of the chunk being finished (residual launches)
    uint32_t cur_parity = 0;
    auto issue_residual = [&]() {
      int mt, col;
      if (!cursor_next(ld, mt, col)) return;
      const int slot = ld_slot;
      if (++ld_slot == slots) ld_slot = 0;
      mbar_expect_tx(&res_bar[ew][slot], 32u * (kHalf ? 64u : 128u));   // rows of 32 bfloat16 or fp32
      if (kMode == kModeRows) {
        tma_load_3d(&map_res, &res_bar[ew][slot], slot_ptr(slot), col, seg_start(mt) + quad * 32, row_of(mt));
      } else {
        tma_load_3d(&map_res, &res_bar[ew][slot], slot_ptr(slot), col, mt * kBlockM + quad * 32, 0);
      }
    };
    // Residual sub-tiles are requested `res_depth` chunks ahead: a request takes
    // a DRAM round trip (one to two microseconds), several times the time a warp
    // needs per chunk.  Requesting chunk g + depth reuses the slot of chunk
    // g + depth - slots, so at most slots - depth - 1 of the latest stores may
    // still be reading shared memory at that point.
    const int res_depth = args.res_depth;
    const int stores_in_flight = slots - res_depth - 1;
    if (kStaged && has_res && lane == 0) {
      for (int d = 0; d < res_depth; ++d) issue_residual();
    }


    int seq = 0;                         // chunks this warp has finished
    int local = 0;
    bool alive = true;
    MCB200_TRACE_DECL;
    MCB200_TRACE_CHUNK_DECL;
    // The first chunk once over before there is anything to read (`dry`: nothing is waited for, stored or handed
    // back): these warps have nothing else to do until the first accumulator is full, and the code they run then comes
    // out of the instruction caches.  Per pass, input resident, ResNet-50 with one image 387 -> 379 us, batch 64 1833 -> 1820.
    // Not with a residual, whose arrival it would wait for first: 256 -> 1024 and a residual at 14 x 14, two images in bfloat16,
    // 5.4 us with and 4.3 without, ResNet-50 with these two images 360 -> 355 us.
    bool dry = !kStaged && !has_res;
    for (int tile = worker; !kSplit && tile < num_tiles && alive; tile += dry ? 0 : workers, local += dry ? 0 : 1, dry = false) {
      const int ab = accumulators == 2 ? local & 1 : 0;
      const uint32_t use = static_cast<uint32_t>(accumulators == 2 ? local >> 1 : local) & 1u;
      // Where the tile lies, before the wait: the divisions cost a few hundred cycles.
      const int unit = tile / n_tiles;
      const int n0 = kMode == kModePhase ? tile_n0(tile) : (tile - unit * n_tiles) * BN;
      int box_row = unit_to_mt(unit), box_image = 0;   // staged form: first output row of this warp's boxes
      if (kMode == kModeRows) {
        box_image = row_of(box_row);
        box_row = (box_row - box_image * args.row_segments) * args.tile_rows + quad * 32;
      } else {
        box_row = box_row * kBlockM + quad * 32;
      }
      // tcgen05.ld is warp-collective: the whole warp takes the same branch.
      if (!dry) alive = __all_sync(0xffffffffu, mbar_wait_bounded(&tmem_full_bar[ab], use, abort, wait_limit));
      if (!alive) break;
      tc_fence_after_sync();
      if (ew == 0 && lane == 0) MCB200_TRACE(3);
      // Per-column constants of the tile's columns go to shared memory.  Two
      // copies (tile parity), each kept while the CTA's tiles of that parity stay
      // in the same column range (always, when the layer has one N tile or the
      // grid is a multiple of the N tiles).  A copy may be overwritten here: the
      // accumulator of this parity is full again, so every warp has read what it
      // needed for the tile that last used the copy.
      const float* t_scale = col_scale[ab];
      const float* t_shift = col_shift[ab];
      const float* t_slope = col_slope[ab];
      const bool refill = table_n0[ab] != n0;
      if (refill) fill_table(ab, n0);
      if (!dry && (refill || local == 0)) {
        // Rendezvous of the epilogue warps on the table (an mbarrier rather than a
        // named barrier, so that the wait is bounded like every other one).
        alive = __all_sync(0xffffffffu, mbar_wait_bounded(&col_bar[ab], table_fills[ab] & 1u, abort, wait_limit));
        if (!alive) break;
        ++table_fills[ab];
      }
      const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(ab * acc_columns) + (static_cast<uint32_t>(quad * 32) << 16);
      const int next = tile + workers;
      int next_rows[4] = {rows[0], rows[1], rows[2], rows[3]};   // (behind the last tile they are not used)
      if (dry) rows[0] = rows[1] = rows[2] = rows[3] = -1;
      // After the last read of this accumulator (and of the per-column tables) it goes back to the MMA
      // issuer, and the next tile's first residual is asked for.
      auto hand_back = [&]() {
        if (dry) return;
        if (ew == 0 && lane == 0) MCB200_TRACE(3);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (kPair) {
            mbar_arrive_cluster(tmem_empty_leader + static_cast<uint32_t>(ab) * 8u);
          } else {
            mbar_arrive(&tmem_empty_bar[ab]);
          }
        }
        if (!kStaged && next < num_tiles) {
          tile_rows(next, next_rows);
          if (has_res) fetch_residual(next_rows, tile_n0(next) + half * kChunk);
        }
      };
      bool handed = false;
#pragma unroll 1
      for (int chunk = half; kStaged && chunk < kChunks; chunk += 2) {
        const int col0 = n0 + chunk * 32;
        if (col0 >= args.cout) break;          // uniform across the warp
        const int g = seq++;
        uint32_t acc[32];
        MCB200_TRACE_CHUNK();
        tmem_load_32x32(tmem_acc + static_cast<uint32_t>(chunk * 32), acc);
        tmem_load_wait();
        MCB200_TRACE_CHUNK();
        const float4* sc4 = reinterpret_cast<const float4*>(t_scale + chunk * 32);
        const float4* sh4 = reinterpret_cast<const float4*>(t_shift + chunk * 32);
        const float4* sl4 = reinterpret_cast<const float4*>(t_slope + chunk * 32);
        // v = acc * scale + shift (+ coeff * residual), then the activation.  The
        // activation is a compile-time tag: with a run-time test inside, every
        // group of four values became its own chain of small basic blocks (load,
        // multiply-add, branch, ...), each exposing its latencies, and a sub-tile
        // took over a thousand cycles; as straight-line code the 32 chains of a
        // row overlap.
        auto finish4 = [&](auto act_tag, int j, float4 r, bool add_res) {
          constexpr int kAct = decltype(act_tag)::value;
          const float4 sc = sc4[j], sh = sh4[j];
          float4 v;
          v.x = fmaf(__uint_as_float(acc[j * 4 + 0]), sc.x, sh.x);
          v.y = fmaf(__uint_as_float(acc[j * 4 + 1]), sc.y, sh.y);
          v.z = fmaf(__uint_as_float(acc[j * 4 + 2]), sc.z, sh.z);
          v.w = fmaf(__uint_as_float(acc[j * 4 + 3]), sc.w, sh.w);
          if (add_res) {
            v.x = fmaf(ep.residual_coeff, r.x, v.x);
            v.y = fmaf(ep.residual_coeff, r.y, v.y);
            v.z = fmaf(ep.residual_coeff, r.z, v.z);
            v.w = fmaf(ep.residual_coeff, r.w, v.w);
          }
          if (kAct == 1) {
            v.x = fmaxf(v.x, 0.f);
            v.y = fmaxf(v.y, 0.f);
            v.z = fmaxf(v.z, 0.f);
            v.w = fmaxf(v.w, 0.f);
          } else if (kAct == 2) {
            const float4 sl = sl4[j];
            v.x = v.x > 0.f ? v.x : v.x * sl.x;
            v.y = v.y > 0.f ? v.y : v.y * sl.y;
            v.z = v.z > 0.f ? v.z : v.z * sl.z;
            v.w = v.w > 0.f ? v.w : v.w * sl.w;
          }
          return v;
        };
        auto round4 = [&](float4& v) {
          v.x = round_to_tf32(v.x);
          v.y = round_to_tf32(v.y);
          v.z = round_to_tf32(v.z);
          v.w = round_to_tf32(v.w);
        };
        const int slot = has_res ? cur_slot : (slots == 2 ? (g & 1) : 0);
        float* buf = slot_ptr(slot) + lane * 32;
        if (has_res) {
          if (lane == 0) {
            switch (stores_in_flight) {
              case 0: tma_store_wait_read<0>(); break;
              case 1: tma_store_wait_read<1>(); break;
              case 2: tma_store_wait_read<2>(); break;
              default: tma_store_wait_read<3>(); break;
            }
            issue_residual();
          }
          alive = __all_sync(0xffffffffu,
                             mbar_wait_bounded(&res_bar[ew][slot], cur_parity, abort, wait_limit));
          if (!alive) break;
          if (++cur_slot == slots) {
            cur_slot = 0;
            cur_parity ^= 1u;
          }
        }
        MCB200_TRACE_CHUNK();
        // Row `lane` of the 32 x 32 tile is 128 bytes: eight 16-byte pieces,
        // piece j stored at position j ^ (row & 7) (the 128-byte swizzle).
        // The result overwrites the residual in place.
        const int swz = lane & 7;
        // All reads of the chunk (residual cells, per-column tables) come
        // before its first write: the loads are then independent of each other
        // and overlap, where a read-modify-write per cell would expose one
        // shared-memory round trip after the other (long ones while the
        // tensor core and the TMA keep shared memory busy).
        float4 v[8];
        // bfloat16 rows are 64 bytes: four 16-byte pieces, piece q stored at
        // position q ^ ((row >> 1) & 3) (the 64-byte swizzle).
        uint8_t* hrow = reinterpret_cast<uint8_t*>(slot_ptr(slot)) + lane * 64;
        const int hswz = (lane >> 1) & 3;
        auto fill = [&](auto act_tag) {
          if (!has_res) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = finish4(act_tag, j, make_float4(0.f, 0.f, 0.f, 0.f), false);
          } else if (kHalf) {
            uint4 w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = *reinterpret_cast<const uint4*>(hrow + ((q ^ hswz) << 4));
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              v[2 * q] = finish4(act_tag, 2 * q,
                                 make_float4(bf16_lo(w[q].x), bf16_hi(w[q].x), bf16_lo(w[q].y), bf16_hi(w[q].y)), true);
              v[2 * q + 1] = finish4(act_tag, 2 * q + 1,
                                     make_float4(bf16_lo(w[q].z), bf16_hi(w[q].z), bf16_lo(w[q].w), bf16_hi(w[q].w)),
                                     true);
            }
          } else {
            float4 r[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = *reinterpret_cast<const float4*>(buf + ((j ^ swz) << 2));
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = finish4(act_tag, j, r[j], true);
          }
        };
        const int act = (kTwo && col0 >= args.second_begin) ? args.second_act : act_mode;
        if (act == 1) {
          fill(Tag<1>());
        } else if (act == 0) {
          fill(Tag<0>());
        } else {
          fill(Tag<2>());
        }
        if (ep.round_tf32) {
#pragma unroll
          for (int j = 0; j < 8; ++j) round4(v[j]);
        }
        if (!has_res && g >= slots) {
          // The store that last used this slot must have finished reading it.  Asked only now,
          // with the chunk's values in registers: the query costs its thread some 200 cycles
          // whatever the answer, which the table loads above spend in flight.
          if (lane == 0) {
            if (slots == 2) {
              tma_store_wait_read<1>();
            } else {
              tma_store_wait_read<0>();
            }
          }
          __syncwarp();
        }
        // Residual and result rows of different widths overlap other lanes' rows.
        if (has_res && (args.out_half != 0) != kHalf) __syncwarp();
        if (args.out_half) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 w;
            w.x = pack_bf16x2(v[2 * q].x, v[2 * q].y);
            w.y = pack_bf16x2(v[2 * q].z, v[2 * q].w);
            w.z = pack_bf16x2(v[2 * q + 1].x, v[2 * q + 1].y);
            w.w = pack_bf16x2(v[2 * q + 1].z, v[2 * q + 1].w);
            *reinterpret_cast<uint4*>(hrow + ((q ^ hswz) << 4)) = w;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) *reinterpret_cast<float4*>(buf + ((j ^ swz) << 2)) = v[j];
        }
        MCB200_TRACE_CHUNK();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // clipped at the row's (the matrix's) end; a launch of two layers has no residual
          if ((kTwo && col0 >= args.second_begin)) {
            tma_store_3d(&map_res, slot_ptr(slot), col0 - args.second_begin, box_row, box_image);
          } else {
            tma_store_3d(&map_out, slot_ptr(slot), col0, box_row, box_image);
          }
          tma_store_commit();
        }
        MCB200_TRACE_CHUNK();
      }
#pragma unroll 1
      for (int chunk = half; !kStaged && chunk < kChunks; chunk += 2) {
        const int col0 = n0 + chunk * kChunk;
        if (col0 >= args.cout) break;          // uniform across the warp
        uint32_t acc[2][4 * kGroups];          // lanes 0-15 and 16-31 of the quadrant
        MCB200_TRACE_CHUNK();
        tmem_load_16x256<kGroups>(tmem_acc + static_cast<uint32_t>(chunk * kChunk), acc[0]);
        if (row_sets > 2) tmem_load_16x256<kGroups>(tmem_acc + (16u << 16) + static_cast<uint32_t>(chunk * kChunk), acc[1]);
        tmem_load_wait();
        // The segments' sums, first to last: the order in which a cluster that splits the tile adds them.
#pragma unroll 1
        for (int i = 1; kSegments && i < segments; ++i) {
          uint32_t more[2][4 * kGroups];
          const uint32_t at = tmem_acc + static_cast<uint32_t>(i * BN + chunk * kChunk);
          tmem_load_16x256<kGroups>(at, more[0]);
          if (row_sets > 2) tmem_load_16x256<kGroups>(at + (16u << 16), more[1]);
          tmem_load_wait();
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 4 * kGroups; ++k)
              acc[h][k] = __float_as_uint(__fadd_rn(__uint_as_float(acc[h][k]), __uint_as_float(more[h][k])));
        }
        MCB200_TRACE_CHUNK();
        // Which layer's columns these are.
        const bool second = (kTwo && col0 >= args.second_begin);
        const int act = second ? args.second_act : act_mode;
        float* const out = second ? args.second_out : args.out;
        const int out_ld = second ? args.second_ld : args.out_ld;
        const int side0 = second ? col0 - args.second_begin : col0;
        const int side_cout = second ? args.cout - args.second_begin : args.first_cout;
        // v = acc * scale + shift (+ coeff * residual), then the activation, in place.  Activation and
        // residual are compile-time tags: with run-time tests inside, every value became its own chain of
        // small basic blocks, each exposing its latencies; as straight-line code the chains overlap.
        auto finish = [&](auto act_tag, auto res_tag) {
          constexpr int kAct = decltype(act_tag)::value;
          constexpr bool kRes = decltype(res_tag)::value != 0;
#pragma unroll
          for (int j = 0; j < kGroups; ++j) {
            const int at = chunk * kChunk + 8 * j + col_in;
            const float2 sc = *reinterpret_cast<const float2*>(t_scale + at);
            const float2 sh = *reinterpret_cast<const float2*>(t_shift + at);
            float2 sl = make_float2(0.f, 0.f);
            if (kAct == 2) sl = *reinterpret_cast<const float2*>(t_slope + at);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (i >= row_sets) break;
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                uint32_t& cell = acc[i >> 1][4 * j + 2 * (i & 1) + e];
                float v = fmaf(__uint_as_float(cell), e ? sc.y : sc.x, e ? sh.y : sh.x);
                if (kRes) v = fmaf(ep.residual_coeff, res[i][j][e], v);
                if (kAct == 1) v = fmaxf(v, 0.f);
                if (kAct == 2) v = v > 0.f ? v : v * (e ? sl.y : sl.x);
                cell = __float_as_uint(v);
              }
            }
          }
        };
        if (has_res) {
          if (act_mode == 1) {
            finish(Tag<1>(), Tag<1>());
          } else if (act_mode == 0) {
            finish(Tag<0>(), Tag<1>());
          } else {
            finish(Tag<2>(), Tag<1>());
          }
        } else if (act == 1) {
          finish(Tag<1>(), Tag<0>());
        } else if (act == 0) {
          finish(Tag<0>(), Tag<0>());
        } else {
          finish(Tag<2>(), Tag<0>());
        }
        if (ep.round_tf32) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 4 * kGroups; ++k) acc[h][k] = __float_as_uint(round_to_tf32(__uint_as_float(acc[h][k])));
        }
        MCB200_TRACE_CHUNK();
        if (chunk + 2 >= kChunks || col0 + 2 * kChunk >= args.cout) {
          hand_back();
          handed = true;
        } else if (has_res && !dry) {
          fetch_residual(rows, col0 + 2 * kChunk);
        }
        MCB200_TRACE_CHUNK();
        if (vec && !args.out_half) {
          // Four lanes hold 32 bytes of a row: a store instruction writes eight whole sectors.
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (i >= row_sets || rows[i] < 0) continue;
            float* dst = out + static_cast<size_t>(rows[i]) * out_ld + side0 + col_in;
#pragma unroll
            for (int j = 0; j < kGroups; ++j) {
              if (side0 + 8 * j + col_in < side_cout)
                *reinterpret_cast<float2*>(dst + 8 * j) =
                    make_float2(__uint_as_float(acc[i >> 1][4 * j + 2 * (i & 1)]), __uint_as_float(acc[i >> 1][4 * j + 2 * (i & 1) + 1]));
            }
          }
        } else if (vec) {
          // As bfloat16 a lane's two columns are one word; the four lanes of a row exchange theirs (a 4 x 4
          // transpose) so that each stores eight columns, 16 bytes.  Word k of a block is group k of one
          // row set, or with two groups per chunk, group k & 1 of two row sets.
          constexpr int kSets = 4 / kGroups;   // row sets in a block
          const int q = lane & 3;
#pragma unroll
          for (int b = 0; b < 4 / kSets; ++b) {
            if (b * kSets >= row_sets) break;
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int i = b * kSets + k / kGroups, j = k % kGroups;
              w[k] = pack_bf16x2(__uint_as_float(acc[i >> 1][4 * j + 2 * (i & 1)]), __uint_as_float(acc[i >> 1][4 * j + 2 * (i & 1) + 1]));
            }
            quad_transpose(w, q);
            int row = rows[b * kSets];
            if (kSets == 2 && q >= 2) row = rows[b * kSets + kSets - 1];
            const int c = side0 + 8 * (q % kGroups);
            if (row >= 0 && c < side_cout)
              *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out) + static_cast<size_t>(row) * out_ld + c) =
                  make_uint4(w[0], w[1], w[2], w[3]);
          }
        } else {
          // Rows whose pitch or start rules wide accesses out, element by element.
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (i >= row_sets || rows[i] < 0) continue;
            const size_t at = static_cast<size_t>(rows[i]) * out_ld + side0 + col_in;
#pragma unroll
            for (int k = 0; k < 2 * kGroups; ++k) {
              const int j = k >> 1, e = k & 1;
              if (side0 + 8 * j + col_in + e >= side_cout) continue;
              const float v = __uint_as_float(acc[i >> 1][4 * j + 2 * (i & 1) + e]);
              if (args.out_half) {
                reinterpret_cast<uint16_t*>(out)[at + 8 * j + e] = static_cast<uint16_t>(pack_bf16x2(v, 0.f));
              } else {
                out[at + 8 * j + e] = v;
              }
            }
          }
        }
        MCB200_TRACE_CHUNK();
        if (dry) break;
      }
      if (!handed) hand_back();   // (staged: the arrival among the chunk's shared-memory writes cost more than it gave, 1 to 2 %)
#pragma unroll
      for (int i = 0; i < 4; ++i) rows[i] = next_rows[i];
    }
    if (kStaged && lane == 0) tma_store_wait_read<0>();
    if (kSplit) {
      // A cluster has one tile.  Each CTA sends every partial sum to the CTA that finishes it: of a chunk's four
      // pieces (its groups of eight columns, or with two groups the upper and lower rows of each) CTA r of the
      // cluster finishes pieces [r, r + 1) * 4 / segments.
      constexpr int kOwn = kChunks > 1 ? kChunks / 2 : 1;   // chunks of a warp
      const int n0 = tile_n0(worker);
      const int pieces = 4 >> args.segment_shift;           // per CTA and chunk
      const int words = kGroups == 4 ? row_sets : row_sets >> 1;   // row sets of a piece
      // Place of a partial sum: [chunk][piece][source][row set][warp][lane], two floats each.
      auto place = [&](int own, int piece, int source, int word) {
        return smem_addr(exchange) +
               8u * static_cast<uint32_t>((((((own * pieces + piece) << args.segment_shift) + source) * words + word) * kEpilogueWarps + ew) * 32 + lane);
      };
      alive = worker < num_tiles && __all_sync(0xffffffffu, mbar_wait_bounded(&tmem_full_bar[0], 0u, abort, wait_limit));
      if (alive) alive = __all_sync(0xffffffffu, mbar_wait_bounded(&col_bar[0], 0u, abort, wait_limit));
      if (alive) {
        tc_fence_after_sync();
#pragma unroll
        for (int own = 0; own < kOwn; ++own) {
          const int chunk = half + 2 * own;
          if (chunk >= kChunks || n0 + chunk * kChunk >= args.cout) break;   // uniform across the warp
          uint32_t acc[2][4 * kGroups];
          const uint32_t at = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(chunk * kChunk);
          tmem_load_16x256<kGroups>(at, acc[0]);
          if (row_sets > 2) tmem_load_16x256<kGroups>(at + (16u << 16), acc[1]);
          tmem_load_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (i >= row_sets) break;
#pragma unroll
            for (int j = 0; j < kGroups; ++j) {
              const int lower = kGroups == 2 && i >= words ? 1 : 0;
              const int piece = kGroups == 4 ? j : 2 * j + lower;
              const int owner = piece >> (2 - args.segment_shift);
              cluster_store(cluster_map(place(own, piece - owner * pieces, static_cast<int>(split_rank), i - lower * words),
                                        static_cast<uint32_t>(owner)),
                            __uint_as_float(acc[i >> 1][4 * j + 2 * (i & 1)]), __uint_as_float(acc[i >> 1][4 * j + 2 * (i & 1) + 1]));
            }
          }
        }
      }
      // The partial sums are where they are finished (a CTA that gave up is here too: its status says so).
      __syncwarp();
      cluster_sync_all();
#pragma unroll 1
      for (int own = 0; alive && own < kOwn; ++own) {
        const int chunk = half + 2 * own;
        const int col0 = n0 + chunk * kChunk;
        if (chunk >= kChunks || col0 >= args.cout) break;
#pragma unroll 1
        for (int piece = 0; piece < pieces; ++piece) {
          const int which = static_cast<int>(split_rank) * pieces + piece;
          const int lower = kGroups == 2 ? which & 1 : 0;
          const int in_chunk = 8 * (kGroups == 4 ? which : which >> 1) + col_in;
          const bool second = (kTwo && col0 >= args.second_begin);
          const int act = second ? args.second_act : act_mode;
          float* const out = second ? args.second_out : args.out;
          const int out_ld = second ? args.second_ld : args.out_ld;
          const int side_cout = second ? args.cout - args.second_begin : args.first_cout;
          const int c = (second ? col0 - args.second_begin : col0) + in_chunk;
          const float2 sc = *reinterpret_cast<const float2*>(&col_scale[0][chunk * kChunk + in_chunk]);
          const float2 sh = *reinterpret_cast<const float2*>(&col_shift[0][chunk * kChunk + in_chunk]);
          const float2 sl = *reinterpret_cast<const float2*>(&col_slope[0][chunk * kChunk + in_chunk]);
#pragma unroll
          for (int word = 0; word < 4; ++word) {
            if (word >= words) break;
            const int row = kGroups == 4 ? rows[word] : lower == 0 ? rows[word & 1] : rows[(word + words) & 3];
            float v[2] = {0.f, 0.f};
#pragma unroll
            for (int source = 0; source < 4; ++source) {
              if (source >= segments) break;
              const float2 part = *reinterpret_cast<const float2*>(exchange + (place(own, piece, source, word) - smem_addr(exchange)));
              v[0] = source == 0 ? part.x : __fadd_rn(v[0], part.x);
              v[1] = source == 0 ? part.y : __fadd_rn(v[1], part.y);
            }
            if (row < 0 || c >= side_cout) continue;
            const bool second = c + 1 < side_cout;
            const size_t at = static_cast<size_t>(row) * out_ld + c;
            v[0] = fmaf(v[0], sc.x, sh.x);
            v[1] = fmaf(v[1], sc.y, sh.y);
            if (has_res) {
              const size_t r = static_cast<size_t>(row) * ep.residual_ld + c;
              const uint16_t* narrow = reinterpret_cast<const uint16_t*>(ep.residual);
              v[0] = fmaf(ep.residual_coeff, kHalf ? bf16_lo(narrow[r]) : ep.residual[r], v[0]);
              if (second) v[1] = fmaf(ep.residual_coeff, kHalf ? bf16_lo(narrow[r + 1]) : ep.residual[r + 1], v[1]);
            }
            if (act == 1) {
              v[0] = fmaxf(v[0], 0.f);
              v[1] = fmaxf(v[1], 0.f);
            } else if (act == 2) {
              v[0] = v[0] > 0.f ? v[0] : v[0] * sl.x;
              v[1] = v[1] > 0.f ? v[1] : v[1] * sl.y;
            }
            if (ep.round_tf32) {
              v[0] = round_to_tf32(v[0]);
              v[1] = round_to_tf32(v[1]);
            }
            if (args.out_half) {
              uint16_t* dst = reinterpret_cast<uint16_t*>(out) + at;
              const uint32_t w = pack_bf16x2(v[0], v[1]);
              if (vec) {
                *reinterpret_cast<uint32_t*>(dst) = w;
              } else {
                dst[0] = static_cast<uint16_t>(w);
                if (second) dst[1] = static_cast<uint16_t>(w >> 16);
              }
            } else if (vec) {
              *reinterpret_cast<float2*>(out + at) = make_float2(v[0], v[1]);
            } else {
              out[at] = v[0];
              if (second) out[at + 1] = v[1];
            }
          }
        }
      }
    }
    __syncwarp();
  }

  if (kSplit && warp < kFirstEpilogueWarp) {
    __syncwarp();
    cluster_sync_all();   // the other warps' is between their sending and finishing
  }

  // ------------------------------------------------------------ teardown
  // A pair leaves together: until both CTAs are here, the peer may still
  // signal this CTA's barriers or (rank 0's MMAs) write its tensor memory.
  tc_fence_before_sync();
  __syncwarp();
  if (kPair) {
    cluster_sync_all();
  } else {
    __syncthreads();
  }
  if (warp == kWarpMma) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, static_cast<uint32_t>(accumulators * acc_columns));
  }
  if (threadIdx.x == 0 && abort_flag && args.status) *static_cast<volatile int*>(args.status) = 1;
}

// ------------------------------------------------------------------ weight packing

__global__ void pack_weights_kernel(const float* __restrict__ w, float* __restrict__ packed, int cout, int c, int taps,
                                    int c_pad) {
  const size_t total = static_cast<size_t>(cout) * taps * c_pad;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int cc = static_cast<int>(i % c_pad);
    const int tap = static_cast<int>((i / c_pad) % taps);
    const int co = static_cast<int>(i / (static_cast<size_t>(c_pad) * taps));
    float v = 0.f;
    if (cc < c) v = round_to_tf32(w[(static_cast<size_t>(co) * c + cc) * taps + tap]);
    packed[i] = v;
  }
}

// Same image in bfloat16 (round to nearest even), taps padded to a multiple of 64 channels.
__global__ void pack_weights_bf16_kernel(const float* __restrict__ w, uint16_t* __restrict__ packed, int cout, int c,
                                         int taps, int c_pad) {
  const size_t total = static_cast<size_t>(cout) * taps * c_pad;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int cc = static_cast<int>(i % c_pad);
    const int tap = static_cast<int>((i / c_pad) % taps);
    const int co = static_cast<int>(i / (static_cast<size_t>(c_pad) * taps));
    float v = 0.f;
    if (cc < c) v = w[(static_cast<size_t>(co) * c + cc) * taps + tap];
    packed[i] = static_cast<uint16_t>(pack_bf16x2(v, 0.f));
  }
}

// fp32 <-> bfloat16 copies of an activation tensor (the layout does not change).
__global__ void f32_to_bf16_kernel(const float4* __restrict__ src, uint2* __restrict__ dst, size_t quads,
                                   const float* __restrict__ src1, uint16_t* __restrict__ dst1, size_t count) {
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  const size_t first = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  for (size_t i = first; i < quads; i += stride) {
    const float4 v = src[i];
    dst[i] = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
  }
  for (size_t i = quads * 4 + first; i < count; i += stride) dst1[i] = static_cast<uint16_t>(pack_bf16x2(src1[i], 0.f));
}

__global__ void bf16_to_f32_kernel(const uint2* __restrict__ src, float4* __restrict__ dst, size_t quads,
                                   const uint16_t* __restrict__ src1, float* __restrict__ dst1, size_t count) {
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  const size_t first = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  for (size_t i = first; i < quads; i += stride) {
    const uint2 w = src[i];
    dst[i] = make_float4(bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y));
  }
  for (size_t i = quads * 4 + first; i < count; i += stride)
    dst1[i] = __uint_as_float(static_cast<uint32_t>(src1[i]) << 16);
}

// ------------------------------------------------------------------ grouped layers

// Grouped layers run with 64-column N tiles (the narrowest: the fewest foreign channels under a
// tile's weight columns).  First channel an N tile's weight columns refer to, and how many
// channel blocks the widest tile spans.
constexpr int kGroupedBlockN = 64;

__host__ __device__ inline int grouped_origin(int n0, int group_cout, int group_cin, int align) {
  return ((n0 / group_cout) * group_cin) & ~(align - 1);
}

int grouped_c_blocks(const mcb200_conv_shape* s, int kelems, int align) {
  const int group_cout = s->cout / s->group, group_cin = s->c / s->group;
  int widest = 0;
  for (int n0 = 0; n0 < s->cout; n0 += kGroupedBlockN) {
    const int last = (n0 + kGroupedBlockN < s->cout ? n0 + kGroupedBlockN : s->cout) - 1;
    const int span = (last / group_cout + 1) * group_cin - grouped_origin(n0, group_cout, group_cin, align);
    if (span > widest) widest = span;
  }
  return (widest + kelems - 1) / kelems;
}

// Packed image of grouped weights [cout][cin / group][taps]: [cout][taps][c_pad] where column j of
// an output channel's row stands for input channel origin(tile of the output channel) + j; zero
// where that channel belongs to another group (or lies beyond the tensor).
template <bool kHalf>
__global__ void pack_weights_grouped_kernel(const float* __restrict__ w, void* __restrict__ packed_any, int cout, int taps,
                                            int c_pad, int group_cout, int group_cin) {
  const size_t total = static_cast<size_t>(cout) * taps * c_pad;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int j = static_cast<int>(i % c_pad);
    const int tap = static_cast<int>((i / c_pad) % taps);
    const int co = static_cast<int>(i / (static_cast<size_t>(c_pad) * taps));
    const int origin = grouped_origin(co / kGroupedBlockN * kGroupedBlockN, group_cout, group_cin, kHalf ? 8 : 4);
    const int local = origin + j - (co / group_cout) * group_cin;   // channel index inside co's group
    float v = 0.f;
    if (local >= 0 && local < group_cin) v = w[(static_cast<size_t>(co) * group_cin + local) * taps + tap];
    if (kHalf) {
      static_cast<uint16_t*>(packed_any)[i] = static_cast<uint16_t>(pack_bf16x2(v, 0.f));
    } else {
      static_cast<float*>(packed_any)[i] = round_to_tf32(v);
    }
  }
}

// ------------------------------------------------------------------ tensor maps

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const int*, const int*, cuuint32_t, cuuint32_t,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct DriverApi {
  EncodeTiledFn tiled = nullptr;
  EncodeIm2colFn im2col = nullptr;
  int driver_version = 0;
  bool ok = false;
};

const DriverApi& driver_api() {
  static DriverApi api;
  static std::once_flag once;
  std::call_once(once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess || !fn)
      return;
    api.tiled = reinterpret_cast<EncodeTiledFn>(fn);
    fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess || !fn)
      return;
    api.im2col = reinterpret_cast<EncodeIm2colFn>(fn);
    cudaDriverGetVersion(&api.driver_version);
    api.ok = true;
  });
  return api;
}

// Tile width.  The kernel is persistent (one CTA per SM), so a layer takes as
// long as its busiest CTA: ceil(tiles / SMs) tiles, each costing its k-iterations
// (operand bytes per iteration grow with BN) plus an epilogue proportional to BN.
// Wide tiles re-read the activations less often, narrow tiles fill the machine
// when there are few output pixels; take the cheapest of the three.
int pick_block_n(int cout, long long m, int k_iters, int widest) {
  const char* force = getenv("MCB200_BLOCK_N");   // "64" / "128" / "256": override for experiments and tests
  if (force) {
    const int bn = atoi(force);
    if (bn == 64 || bn == 128 || bn == 256) return bn;
  }
  const long long m_tiles = (m + kBlockM - 1) / kBlockM;
  int best = 64;
  double best_cost = 0.0;
  for (int bn = 64; bn <= widest; bn *= 2) {
    if (bn > 64 && bn / 2 >= cout) break;   // wider than the layer: only padding
    const long long tiles = m_tiles * ((cout + bn - 1) / bn);
    const long long waves = (tiles + 147) / 148;
    // 64 KiB of operand-byte equivalents per 32-column chunk of epilogue: a chunk costs a warp
    // 1400-2300 cycles (two warps per tensor-memory quadrant), as long as some 64 KiB take to
    // arrive.  (Measured in interleaved runs of the three benchmark networks: the 8 KiB this
    // started with sent the 128 -> 512 residual layers of ResNet-50 to 256-column tiles, six waves
    // of eight chunks where eleven waves of four are 6 % quicker; values of 48-96 KiB agree.)
    const double per_tile = static_cast<double>(k_iters) * (kTileABytes + 128.0 * bn) + 65536.0 * (bn / 32);
    const double cost = static_cast<double>(waves) * per_tile;
    if (bn == 64 || cost < best_cost * 0.97) {   // prefer the narrower tile on near ties
      best = bn;
      best_cost = cost;
    }
  }
  return best;
}

// Shared memory a CTA can give to the operand ring, roughly (the exact figure depends on the
// kernel variant's static shared memory; the launch computes it).
constexpr int kRingBudget = kSharedLimit - 10 * 1024;

// Halo mode: tile width, pairing and cost by the same model (a CTA's time is its operand bytes).
// A stage holds the pixel strip and the weight tiles of the kw taps of a filter row; widths whose
// stage does not fit three times are left out.  Returns 0 when no width is usable.
int pick_block_n_halo(int cout, long long m_virtual, int k_iters, int kw, int strip_bytes, int* pair_out,
                      double* cost_out) {
  const char* force = getenv("MCB200_BLOCK_N");
  const int forced = force ? atoi(force) : 0;
  const char* force_pair = getenv("MCB200_CTA_PAIR");
  const long long m_tiles = (m_virtual + kBlockM - 1) / kBlockM;
  const int strip_slot = (strip_bytes + 1023) / 1024 * 1024;
  int best = 0;
  double best_cost = 0.0;
  // 256-column tiles only when asked for: on every halo-mode layer measured with both widths
  // (VGG-16 at 300 x 300, batch 32: 256 -> 256 on 75 x 75 maps, 256 -> 512 and 512 -> 512 on 38 x 38;
  // ResNet-50's 512 -> 512 on 7 x 7) paired 128-column tiles are as quick or quicker, by up to 13 %:
  // these layers run near the tensor pipe's rate, where twice as many narrower tiles fill the
  // last wave better and a stage is 41 KiB instead of 65.
  const int widest = forced == 256 ? 256 : 128;
  for (int bn = 64; bn <= widest; bn *= 2) {
    if (bn > 64 && bn / 2 >= cout) break;
    if ((forced == 64 || forced == 128 || forced == 256) && bn != forced) continue;
    for (int pair = 0; pair <= 1; ++pair) {
      if (pair && (bn < 128 || m_tiles < 2)) continue;
      if (force_pair && (force_pair[0] == '0' || force_pair[0] == '1') && bn >= 128 && pair != force_pair[0] - '0')
        continue;
      const int stage = strip_slot + kw * (pair ? bn / 2 : bn) * 128;
      if (kRingBudget / stage < 3) continue;
      const long long units = pair ? (m_tiles + 1) / 2 : m_tiles;
      const long long tiles = units * ((cout + bn - 1) / bn);
      const long long workers = pair ? 74 : 148;
      const long long waves = (tiles + workers - 1) / workers;
      // the pair's cluster-wide synchronisation costs about two k-iterations per tile
      const double per_tile = static_cast<double>(k_iters + (pair ? 2 : 0)) * stage + 8192.0 * (bn / 32);
      const double cost = static_cast<double>(waves) * per_tile;
      if (best == 0 || cost < best_cost * 0.97) {
        best = bn;
        best_cost = cost;
        *pair_out = pair;
      }
    }
  }
  if (cost_out) *cost_out = best_cost;
  return best;
}

// Whether two-CTA clusters run the layer.  Pairing halves the weight bytes each
// SM pulls per MAC, which pays where the operand ring bounds the main loop (wide
// tiles, long K) and there are at least two M tiles to pair up.  Short-K layers
// are bound by their epilogue and only pay for the pair's extra synchronisation
// (measured on ResNet-50: gains from 16 k-iterations up when no residual is
// added, losses at 4-16 with one).
int pick_cta_pair(int block_n, long long m, int k_iters) {
  const char* force = getenv("MCB200_CTA_PAIR");   // "0" / "1": override for experiments
  if (force && (force[0] == '0' || force[0] == '1')) return block_n >= 128 && force[0] == '1' ? 1 : 0;
  // 256-column tiles pair from 16 k-iterations (the 512 -> 1024 stride-2 projection of ResNet-50:
  // 39 -> 34 us), 128-column tiles from 17 (the 512 -> 2048 residual layers lose 1-2 us at 16).
  return (block_n >= 128 && m > kBlockM && k_iters >= (block_n == 256 ? 16 : 17)) ? 1 : 0;
}

// Segments of the sum over K, as a power of two: each is summed on its own and they are added first to last.  By the
// layer's geometry alone: an image's result must not depend on the batch it runs in.
// Worth it from 128 MMA steps per tap chain on.  Large batches pay: such a tile needs a tensor-memory accumulator per
// segment, so with four segments it is at most 128 columns wide and the tile behind it waits until it is drained.  Hence
// four on maps of at most 64 pixels, and up to 256 pixels from 256 steps; else two (256 columns, as without).
// Measured, four / two / one segments: 3 x 3 at 256 channels on 14 x 14, batch 64 39.4 / 35.3 / 35.2 us, ResNet-50 with
// one image 397 / 411 / 454 us per pass; 1024 -> 256 on 14 x 14, batch 64 29.2 / 25.1 / 25.0; 3 x 3 at 512 channels on
// 19 x 19, batch 32 84 / 78 / 78, one image in bfloat16 18.5 / 20.4 / 28.7.
int segment_shift_of(const mcb200_conv_shape& s, int mode, int k_iters) {
  if (s.group != 1 || (mode != kModeMatrix && mode != kModeIm2col && mode != kModeHalo)) return 0;
  const long long steps = static_cast<long long>(k_iters) * (mode == kModeHalo ? s.kw : 1) * kMmaPerBlock;
  const long long positions = static_cast<long long>(s.ho) * s.wo;
  if (positions <= 64) return steps >= 128 ? 2 : 0;
  if (positions <= 256) return steps >= 256 ? 2 : steps >= 128 ? 1 : 0;
  return positions <= 400 && steps >= 512 ? 1 : 0;
}

// CTAs that run at one time as clusters of 1 << shift, one tile each: asked of the device, as a cluster keeps to one GPC and
// how many SMs a GPC has differs from chip to chip (one B200: 74 clusters of two, all 148 SMs, but 33 of four, 132).
// No more than 128 and 144, though: with the thirty-third cluster of four 512 -> 672 channels, 3 x 3, three images of 7 x 7
// gain (11.5 -> 10.2 us) and 2048 -> 1056 on one pixel, which small_tiles then cuts to 32 columns, loses (6.5 -> 7.2).
int split_capacity(int shift) {
  static std::mutex mu;
  static int ctas[64][3] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  std::lock_guard<std::mutex> lock(mu);
  int& known = ctas[dev][shift];
  if (known == 0) {
    auto kernel = conv_tc_kernel<64, kModeMatrix, false, false, kOutSplit>;   // (all forms: one CTA per SM, most of its memory)
    cudaFuncAttributes func;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << shift;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(1u << shift, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncGetAttributes(&func, kernel) == cudaSuccess) {
      cfg.dynamicSmemBytes = static_cast<size_t>(kSharedLimit) - func.sharedSizeBytes;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(cfg.dynamicSmemBytes)) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess)
        clusters = 0;
    }
    if (clusters < 1) {
      (void)cudaGetLastError();
      clusters = 128 >> shift;
    }
    known = std::min(clusters << shift, shift == 2 ? 128 : 144);
  }
  return known;
}

int m_tile_of(const mcb200_conv_plan& p) {
  const int halo_rows = p.im2col == kModeHalo ? (p.shape.kw - 1) * p.shape.dil_w : 0;
  const bool cut = p.im2col == kModeMatrix || p.im2col == kModeIm2col || p.im2col == kModeHalo;
  return cut && p.strip_rows - halo_rows == kSmallM ? kSmallM : kBlockM;
}

int plan_segment_shift(const mcb200_conv_plan& p) {
  int shift = segment_shift_of(p.shape, p.im2col, p.k_iters);
  while ((p.block_n << shift) > 512) --shift;   // a tile width that was asked for (MCB200_BLOCK_N)
  return shift;
}

// Whether a cluster's CTAs make a tile's segments side by side: where all tiles then still run at one time.
bool split_launch(const mcb200_conv_plan& p, int shift) {
  const char* off = getenv("MCB200_SPLIT");   // "0": one CTA makes all segments (experiments and tests)
  if (off && off[0] == '0') return false;
  const long long bm = m_tile_of(p);
  const long long tiles = (p.m_virtual + bm - 1) / bm * ((p.shape.cout + p.block_n - 1) / p.block_n);
  return shift > 0 && !p.cta_pair && p.block_n <= 128 && (tiles << shift) <= split_capacity(shift);
}

// Layers of a single image (or a few) have fewer tiles than the chip has SMs, and the time of one is the chain of its
// k-iterations.  An MMA takes at least 41 cycles with 64 rows and 52 with 128, however few its columns, and the
// copies' writes to shared memory get in the way of its operand reads.  So where the tiles
// all run at once anyway, cut them to 64 pixels and 64 or 32 columns: more SMs, each with a half or a third of the
// bytes per iteration and half the epilogue; and where the sum over K has segments, let a cluster make them side by side.
// The results are the same bits.  Returns whether the layer runs in 64-row tiles, with *block_n and *pair set to match.
// The cost model, in cycles: four MMAs per k-iteration and tap, half of the copies' bytes at 128 per cycle, 1500 per 64
// columns of epilogue, 2000 for the exchange of a split tile.  Only up to one tile per SM: with more, ordinary tiles
// fill the chip; and only for a tenth less by the model, which is no better than that.
// Measured, one image (each launch on its own): 3 x 3 at 256 channels on 14 x 14 18.9 -> 12.8 us, at 512 on 7 x 7
// 27.1 -> 14.8, 2048 -> 1000 classes 18.4 -> 12.3; per pass ResNet-50 496 -> 406, SSD300 in bfloat16 620 -> 495.  (A chip
// that other nets keep busy has no SMs to give.)
bool small_tiles(int cout, long long m, int k_iters, int taps, int halo_rows, int shift, int* block_n, int* pair) {
  const char* force = getenv("MCB200_BLOCK_M");   // "64" / "128": override for experiments and tests
  const bool forced = force && atoi(force) == kSmallM;
  const char* width = getenv("MCB200_BLOCK_N");
  if (forced) {
    *block_n = width && atoi(width) == 32 ? 32 : 64;
    *pair = 0;
    return true;
  }
  if (force || width || getenv("MCB200_CTA_PAIR")) return false;
  auto tiles_of = [&](int bm, int bn) { return ((m + bm - 1) / bm) * ((cout + bn - 1) / bn); };
  auto cost = [&](int bm, int bn, bool paired) {
    const bool split = !paired && shift > 0 && bn <= 128 && (tiles_of(bm, bn) << shift) <= split_capacity(shift);
    const int b_rows = paired ? bn / 2 : bn;
    const double floor = bm == kSmallM ? 40 : 50, pipe = bn / 2.0;
    const double iter = taps * 4 * (pipe > floor ? pipe : floor) + 0.5 * (bm + halo_rows + taps * b_rows);
    return (split ? k_iters >> shift : k_iters) * iter + 1500.0 * ((bn + 63) / 64) + (split ? 2000.0 : 0.0);
  };
  if (tiles_of(kBlockM, *block_n) > 148) return false;
  double best = 0.9 * cost(kBlockM, *block_n, *pair != 0);
  bool small = false;
  for (int bm = kSmallM; bm <= kBlockM; bm *= 2) {
    for (int bn = shift > 0 ? 128 : 64; bn >= 32; bn /= 2) {
      if (tiles_of(bm, bn) > 148 || (bm == kBlockM && shift == 0)) break;
      if (bn > 64 && (bm == kSmallM || bn / 2 >= cout)) continue;
      const double c = cost(bm, bn, false);
      if (c < best) {
        best = c;
        *block_n = bn;
        *pair = 0;
        small = bm == kSmallM;
      }
    }
  }
  return small;
}

// Tile map for the staged epilogue over a row-major matrix with row pitch `ld`
// (elements), boxes of 32 rows x 32 columns: fp32 with the 128-byte swizzle, or bfloat16 (64-byte
// box rows) with the 64-byte swizzle.  The rows are split as (group, row in
// group): ordinary tiles use one group of all rows; row mode uses one group per
// output row of an image so that a tile never spills into the next row.
CUresult encode_tile_map(CUtensorMap* map, const void* base, bool half, int cols, int ld, long long rows_per_group,
                         long long groups) {
  const DriverApi& api = driver_api();
  const cuuint64_t es = half ? 2 : 4;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows_per_group),
                              static_cast<cuuint64_t>(groups)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * es,
                                 static_cast<cuuint64_t>(ld) * es * static_cast<cuuint64_t>(rows_per_group)};
  const cuuint32_t box[3] = {32, 32, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return api.tiled(map, half ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                   const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   half ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

template <int BN, int kMode, bool kPair, bool kHalf, int kOut = kOutDirect>
cudaError_t launch_variant(const mcb200_conv_plan* plan, ConvTcArgs args, cudaStream_t stream) {
  constexpr bool kStaged = kOut == kOutStaged || kOut == kOutStagedTwo, kSplit = kOut == kOutSplit;
  using Plan = SmemPlan<BN, kMode, kPair>;
  auto kernel = conv_tc_kernel<BN, kMode, kPair, kHalf, kOut>;
  // The large-shared-memory opt-in is per device: do it once for each device
  // this process launches on.  What the ring may use is the CTA limit minus the
  // kernel's static shared memory (barriers, per-column tables).
  int dev = 0;
  cudaGetDevice(&dev);
  static bool configured[64] = {false};
  static int sm_count[64] = {0};
  static int dynamic_limit = 0;
  static std::mutex mu;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dynamic_limit == 0) {
      cudaFuncAttributes attr;
      cudaError_t e = cudaFuncGetAttributes(&attr, kernel);
      if (e != cudaSuccess) return e;
      dynamic_limit = kSharedLimit - static_cast<int>(attr.sharedSizeBytes);
    }
    if (dev >= 0 && dev < 64 && !configured[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dynamic_limit);
      if (e != cudaSuccess) return e;
      int n = 0;
      if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
      sm_count[dev] = n;
      configured[dev] = true;
    }
  }
  const long long m_tiles = kMode == kModeRows
                                ? static_cast<long long>(plan->shape.n) * plan->shape.ho * args.row_segments
                                : (static_cast<long long>(args.m) + args.tile_rows - 1) / args.tile_rows;   // halo: virtual positions
  const long long m_units = kPair ? (m_tiles + 1) / 2 : m_tiles;
  const long long n_tiles = kMode == kModePhase
                                ? static_cast<long long>(args.phase_tiles) * args.phase_stride_h * args.phase_stride_w
                                : (plan->shape.cout + BN - 1) / BN;
  const long long tiles = n_tiles * m_units;
  if (tiles > 0x3fffffffLL) return cudaErrorInvalidConfiguration;
  // One persistent CTA per SM (fewer when there are fewer tiles); a paired
  // launch is a grid of two-CTA clusters, one cluster per tile at a time.
  const int sms = (dev >= 0 && dev < 64 && sm_count[dev] > 0) ? sm_count[dev] : 148;
  const long long workers_max = kPair ? sms / 2 : sms;
  const unsigned workers = static_cast<unsigned>(tiles < workers_max ? tiles : workers_max);
  // A stage: sub-tiles of activations, then of weights.
  args.stage_b_offset = Plan::kSub * (args.tile_rows == kSmallM && kMode != kModeRows ? kSmallM : kBlockM) * kBlockK * 4;
  args.stage_bytes = args.stage_b_offset + Plan::kSub * Plan::kTileBBytes;
  int resident_bytes = 0;
  if (kMode == kModeRows) {
    // One N tile: every M tile multiplies the same kh weight tiles; they stay in shared memory
    // when they take at most a quarter of it, and the ring carries activations only.
    const long long all_rows = static_cast<long long>(args.k_iters) * Plan::kTileBBytes;
    const char* off = getenv("MCB200_ROWS_RESIDENT");   // "0": stream the weights with the activations (experiments)
    if (plan->shape.cout <= BN && all_rows <= 56 * 1024 && !(off && off[0] == '0')) resident_bytes = static_cast<int>(all_rows);
    args.resident_b_bytes = resident_bytes;
    if (resident_bytes) args.stage_bytes = args.stage_b_offset;
  }
  if (kMode == kModeHalo) {
    // The pixel strip (rounded up to the 1024-byte swizzle period) + the weight tiles of the kw taps of
    // one filter row.
    args.stage_b_offset = (args.a_bytes + 1023) / 1024 * 1024;
    args.stage_bytes = args.stage_b_offset + plan->shape.kw * Plan::kTileBBytes;
  }
  {
    // At most 64 prefetch instructions per tile (long-K tiles take long enough for the ring).
    const int kh = plan->shape.kh, cb = args.c_blocks;
    const int count = kMode == kModeMatrix ? cb : kh * cb * ((kMode == kModeIm2col && plan->shape.stride_w > 1) ? 2 : 1);
    // Off unless MCB200_L2_PREFETCH=1: measured on ResNet-50 at batch 64 it costs 2 % (the 1 x 1
    // reductions lose 8 %: the requests compete with the loads of the tile at hand), and the
    // layers it was meant for do not gain.
    const char* pf = getenv("MCB200_L2_PREFETCH");
    args.l2_prefetch = (kMode != kModeRows && kMode != kModePhase && count <= 64 && pf && pf[0] == '1') ? 1 : 0;
  }
  int staging_bytes = 0;
  args.slots = args.res_depth = 1;
  if (kStaged) {
    // Slots per epilogue warp.  With a residual three where tiles are so short that the ring needs little (load,
    // work and store of consecutive chunks overlap), else two.  Without: one, and the ring takes the rest.
    if (args.ep.residual != nullptr) args.slots = args.k_iters * (kHalf ? 2 : 1) <= 4 ? 3 : 2;
    staging_bytes = kEpilogueWarps * args.slots * ((kHalf && args.out_half) ? 2048 : 4096);
  }
  if (kSplit) staging_bytes = args.tile_rows * BN * 4;   // as many partial sums arrive at a CTA as its tile has cells
  int stages = (dynamic_limit - 1024 - resident_bytes - staging_bytes) / args.stage_bytes;
  if (stages > kMaxStages) stages = kMaxStages;
  if (stages < 2) return cudaErrorInvalidConfiguration;
  args.stages = stages;
  const int dynamic_bytes = stages * args.stage_bytes + resident_bytes + staging_bytes + 1024;   // + alignment slack
  const CUtensorMap* ma = reinterpret_cast<const CUtensorMap*>(plan->tma_a);
  const CUtensorMap* mb = reinterpret_cast<const CUtensorMap*>(plan->tma_b);
  const CUtensorMap* mo = kStaged ? reinterpret_cast<const CUtensorMap*>(plan->tma_out) : ma;
  const CUtensorMap* mr = kStaged && (args.ep.residual || args.second_out) ? reinterpret_cast<const CUtensorMap*>(plan->tma_res) : ma;
  cudaError_t launched;
  {
    TimedLaunch timed(stream);
    cudaLaunchConfig_t cfg = {};
    const unsigned cluster = kPair ? 2u : kSplit ? 1u << args.segment_shift : 1u;
    cfg.gridDim = dim3((kSplit ? static_cast<unsigned>(tiles) : workers) * cluster, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = static_cast<size_t>(dynamic_bytes);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    // The kernel's set-up may overlap the end of the previous kernel in the
    // stream; it orders itself with griddepcontrol.wait.
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    launched = cudaLaunchKernelEx(&cfg, kernel, *ma, *mb, *mo, *mr, args);
  }
  count_launch();
  return launched;
}

// Whether results leave through shared memory as TMA tiles rather than straight from registers.  Registers are
// the shorter way (a chunk of 32 x 32 takes its warp 1100 cycles, 1400 through shared memory, and the ring gets the
// staging's bytes), which counts where a CTA has one tile whose end nothing overlaps.  But a store
// instruction then writes 32 bytes of eight rows each, and with many tiles in flight that, not HBM, is the limit
// (64 -> 256 columns and a residual on 56 x 56 maps, batch 64: 107 us against 80; 32 -> 64 on 112 x 112, no residual: 71
// against 59), as 16 bytes of a bfloat16 row are.  In fp32, without a residual and with one tile per CTA (three if the
// layer is one tile wide) it is the quicker one for pairs of 128 columns and for no other tile.  Staged and from registers, per
// launch: pairs of 128 columns, 640 -> 512 at 14 x 14, batch 16 10.1 and 9.5 us, 768 -> 128 at 75 x 75, two images 11.0 and 10.1,
// 256 -> 128, 3 x 3 at stride 2, 75 x 75, batch 32 72 and 64; of 256, 768 -> 192 at 24 x 24, batch 32 14.3 and 15.1,
// 640 -> 512 at 38 x 38, four images 13.4 and 14.0; one CTA and 128 columns, 512 -> 512 at 14 x 14, batch 16 7.9 and
// 9.2; 64 columns, 768 -> 512 at 28 x 28, two images 8.3 and 8.7.
bool staged_epilogue(const mcb200_conv_plan* plan, bool residual) {
  const char* force = getenv("MCB200_STAGED");   // "0" / "1": override for experiments and tests
  if (force && (force[0] == '0' || force[0] == '1')) return force[0] == '1';
  const long long m_tiles = plan->im2col == kModeRows
                                ? static_cast<long long>(plan->shape.n) * plan->shape.ho * ((plan->shape.wo + kBlockM - 1) / kBlockM)
                                : (static_cast<long long>(plan->m) + kBlockM - 1) / kBlockM;
  const long long tiles = m_tiles * ((plan->shape.cout + plan->block_n - 1) / plan->block_n);
  const long long workers = plan->cta_pair ? 74 : 148, units = plan->cta_pair ? (tiles + 1) / 2 : tiles;
  const bool one_column = plan->shape.cout <= plan->block_n;
  return residual || plan->operand_bf16 || !plan->cta_pair || plan->block_n != 128 || units > (one_column ? 3 : 1) * workers;
}

}  // namespace
}  // namespace mcb200

using namespace mcb200;

namespace {
// Bound of the kernel's barrier waits (process-wide) and the one-shot test hook of the calling thread.
long long g_wait_limit_cycles = mcb200::kDefaultWaitLimitCycles;
thread_local int t_drop_weight_load = 0;
}  // namespace

namespace mcb200 {
long long conv_wait_limit() { return g_wait_limit_cycles; }
int conv_take_drop_hook() {
  const int drop = t_drop_weight_load;
  t_drop_weight_load = 0;
  return drop;
}
}  // namespace mcb200

extern "C" long long mcb200_conv_set_wait_limit(long long cycles) {
  const long long previous = g_wait_limit_cycles;
  g_wait_limit_cycles = cycles > 0 ? cycles : mcb200::kDefaultWaitLimitCycles;
  return previous;
}

extern "C" void mcb200_conv_test_drop_weight_load(void) { t_drop_weight_load = 1; }

extern "C" int mcb200_conv_out_shape(mcb200_conv_shape* s) {
  if (!s || s->kh < 1 || s->kw < 1 || s->stride_h < 1 || s->stride_w < 1 || s->dil_h < 1 || s->dil_w < 1) return -1;
  const int ext_h = s->dil_h * (s->kh - 1) + 1;
  const int ext_w = s->dil_w * (s->kw - 1) + 1;
  const int num_h = s->h + 2 * s->pad_h - ext_h;
  const int num_w = s->w + 2 * s->pad_w - ext_w;
  if (num_h < 0 || num_w < 0) return -1;
  s->ho = num_h / s->stride_h + 1;
  s->wo = num_w / s->stride_w + 1;
  return 0;
}

extern "C" size_t mcb200_conv_packed_weight_count(const mcb200_conv_shape* s) {
  const size_t c_pad = s->group > 1 ? static_cast<size_t>(grouped_c_blocks(s, kBlockK, 4)) * kBlockK
                                    : static_cast<size_t>((s->c + kBlockK - 1) / kBlockK) * kBlockK;
  return static_cast<size_t>(s->cout) * s->kh * s->kw * c_pad;
}

extern "C" int mcb200_conv_pack_weights(const mcb200_conv_shape* s, const float* w_oihw, float* packed,
                                        void* stream) {
  if (!s || !w_oihw || !packed || s->group < 1 || s->c % s->group != 0 || s->cout % s->group != 0) return -1;
  const size_t total = mcb200_conv_packed_weight_count(s);
  const int threads = 256;
  const int blocks = static_cast<int>((total + threads - 1) / threads < 148 * 8 ? (total + threads - 1) / threads
                                                                                  : 148 * 8);
  if (s->group > 1) {
    pack_weights_grouped_kernel<false><<<blocks > 0 ? blocks : 1, threads, 0, static_cast<cudaStream_t>(stream)>>>(
        w_oihw, packed, s->cout, s->kh * s->kw, grouped_c_blocks(s, kBlockK, 4) * kBlockK, s->cout / s->group,
        s->c / s->group);
    count_launch();
    return static_cast<int>(cudaGetLastError());
  }
  const int c_pad = (s->c + kBlockK - 1) / kBlockK * kBlockK;
  pack_weights_kernel<<<blocks > 0 ? blocks : 1, threads, 0, static_cast<cudaStream_t>(stream)>>>(
      w_oihw, packed, s->cout, s->c, s->kh * s->kw, c_pad);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" size_t mcb200_conv_packed_weight_count_bf16(const mcb200_conv_shape* s) {
  const size_t c_pad = s->group > 1 ? static_cast<size_t>(grouped_c_blocks(s, kBlockKHalf, 8)) * kBlockKHalf
                                    : static_cast<size_t>((s->c + kBlockKHalf - 1) / kBlockKHalf) * kBlockKHalf;
  return static_cast<size_t>(s->cout) * s->kh * s->kw * c_pad;
}

extern "C" int mcb200_conv_pack_weights_bf16(const mcb200_conv_shape* s, const float* w_oihw, uint16_t* packed,
                                             void* stream) {
  if (!s || !w_oihw || !packed || s->group < 1 || s->c % s->group != 0 || s->cout % s->group != 0) return -1;
  const size_t total = mcb200_conv_packed_weight_count_bf16(s);
  const int threads = 256;
  const int blocks = static_cast<int>((total + threads - 1) / threads < 148 * 8 ? (total + threads - 1) / threads
                                                                                  : 148 * 8);
  if (s->group > 1) {
    pack_weights_grouped_kernel<true><<<blocks > 0 ? blocks : 1, threads, 0, static_cast<cudaStream_t>(stream)>>>(
        w_oihw, packed, s->cout, s->kh * s->kw, grouped_c_blocks(s, kBlockKHalf, 8) * kBlockKHalf, s->cout / s->group,
        s->c / s->group);
    count_launch();
    return static_cast<int>(cudaGetLastError());
  }
  const int c_pad = (s->c + kBlockKHalf - 1) / kBlockKHalf * kBlockKHalf;
  pack_weights_bf16_kernel<<<blocks > 0 ? blocks : 1, threads, 0, static_cast<cudaStream_t>(stream)>>>(
      w_oihw, packed, s->cout, s->c, s->kh * s->kw, c_pad);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_f32_to_bf16(const float* src, uint16_t* dst, size_t count, void* stream) {
  if (!src || !dst) return -1;
  if (count == 0) return 0;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) && ((reinterpret_cast<uintptr_t>(dst) & 7) == 0);
  const size_t quads = vec ? count / 4 : 0;
  const size_t items = quads + (count - quads * 4);
  const int blocks = static_cast<int>((items + 255) / 256 < 148 * 16 ? (items + 255) / 256 : 148 * 16);
  f32_to_bf16_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float4*>(src), reinterpret_cast<uint2*>(dst), quads, src, dst, count);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_bf16_to_f32(const uint16_t* src, float* dst, size_t count, void* stream) {
  if (!src || !dst) return -1;
  if (count == 0) return 0;
  const bool vec = ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) && ((reinterpret_cast<uintptr_t>(src) & 7) == 0);
  const size_t quads = vec ? count / 4 : 0;
  const size_t items = quads + (count - quads * 4);
  const int blocks = static_cast<int>((items + 255) / 256 < 148 * 16 ? (items + 255) / 256 : 148 * 16);
  bf16_to_f32_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const uint2*>(src), reinterpret_cast<float4*>(dst), quads, src, dst, count);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

namespace {

// Drivers up to CUDA 13.1 encode a flag in im2col descriptors of tensors smaller than 128 KiB that
// makes the load misbehave; NVIDIA's CUTLASS clears it the same way
// (cute/atom/copy_traits_sm90_im2col.hpp).
void clear_small_tensor_flag(CUtensorMap* map, unsigned long long bytes) {
  if (driver_api().driver_version <= 13010 && bytes < 131072ull) reinterpret_cast<uint64_t*>(map)[1] &= ~(1ull << 21);
}

// Shared by the fp32 (TF32) and the bfloat16 plan: `in` and `packed_w` hold
// elements of `es` bytes, a k-iteration covers `kelems` channels (128 bytes).
int plan_core(const mcb200_conv_shape* s, const void* in, const void* packed_w, mcb200_conv_plan* plan, bool half) {
  const cuuint64_t es = half ? 2 : 4;
  const int kelems = half ? kBlockKHalf : kBlockK;
  const CUtensorMapDataType dtype = half ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  if (!s || !in || !packed_w || !plan) return -1;
  if (s->group < 1 || s->c % s->group != 0 || s->cout % s->group != 0) return -2;
  if ((s->c_stride & (half ? 7 : 3)) != 0 || s->c_stride < s->c) return -2;
  if ((reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(packed_w) & 15)) return -3;
  if (s->pad_h > 127 || s->pad_w > 127 || (s->kh - 1) * s->dil_h > 255 || (s->kw - 1) * s->dil_w > 255) return -4;
  const DriverApi& api = driver_api();
  if (!api.ok) return -5;

  plan->shape = *s;
  plan->out_ptr = nullptr;
  plan->res_ptr = nullptr;
  plan->out_ld = plan->res_ld = plan->cta_pair = 0;
  plan->operand_bf16 = half ? 1 : 0;
  plan->out_bf16 = 0;
  if (mcb200_conv_out_shape(&plan->shape) != 0) return -6;
  const long long m_ll = static_cast<long long>(s->n) * plan->shape.ho * plan->shape.wo;
  if (m_ll <= 0 || m_ll > 0x7fffffffLL) return -7;
  plan->m = static_cast<int>(m_ll);
  const bool grouped = s->group > 1;
  plan->c_blocks = grouped ? grouped_c_blocks(s, kelems, half ? 8 : 4) : (s->c + kelems - 1) / kelems;
  plan->k_iters = s->kh * s->kw * plan->c_blocks;
  const bool pointwise = s->kh == 1 && s->kw == 1 && s->stride_h == 1 && s->stride_w == 1 && s->pad_h == 0 &&
                         s->pad_w == 0;
  const int segments = segment_shift_of(plan->shape, pointwise ? kModeMatrix : kModeIm2col, plan->k_iters);
  plan->block_n = grouped ? kGroupedBlockN : pick_block_n(s->cout, plan->m, plan->k_iters, segments > 1 ? 512 >> segments : 256);
  // The pairing rule was measured in 32-channel k-iterations; a bfloat16 k-iteration covers 64.
  plan->cta_pair = grouped ? 0 : pick_cta_pair(plan->block_n, plan->m, plan->k_iters * (half ? 2 : 1));
  plan->im2col = pointwise ? 0 : 1;
  plan->m_virtual = plan->m;
  plan->strip_rows = 0;
  // Halo mode for stride-1 filters with more than one tap per row: see ConvTcArgs.  The choice
  // depends on the layer's geometry only, never on the batch size: the two modes sum over K in
  // different orders, and an image's result must not depend on how many images run with it.
  // Measured on the benchmark networks (ResNet-50 at batch 64, per 3 x 3 layer): 56-pixel rows
  // 52.8 -> 49.8 us, 28-pixel rows 37.1 -> 33.4, 7-pixel rows 43.0 -> 37.3, but 14-pixel rows 35.3
  // -> 43.3: there every CTA has a single 256-column tile, and the halo mode's epilogue (plain
  // stores, since a tile of the virtual grid is not a box of the output tensor) is exposed where
  // the im2col mode's TMA tile stores are half as long (37.2 against 35.5 us once the mode kept to
  // 128-column tiles).  SSD300 at batch 32, 512 -> 512 on 19-pixel rows: 102 -> 82 us, the two
  // detection heads on the same map 84 -> 69 and 66 -> 63; on its 10-pixel rows 36 -> 38.  Hence:
  // rows of at least 16 output pixels or at most 8 (the strips save the most), and never when the
  // widened rows would cost more than half again as many positions.
  const int halo_w = (s->kw - 1) * s->dil_w;
  const char* halo_env = getenv("MCB200_HALO");   // "0" / "1": override for experiments and tests
  const bool halo_forced = halo_env && halo_env[0] == '1';
  const bool halo_pays = 2 * halo_w <= plan->shape.wo && (plan->shape.wo >= 16 || plan->shape.wo <= 8);
  if (!pointwise && s->stride_h == 1 && s->stride_w == 1 && s->kw > 1 && halo_w <= kMaxHaloRows &&
      !(halo_env && halo_env[0] == '0') && (halo_forced || halo_pays)) {
    const long long mv = static_cast<long long>(s->n) * plan->shape.ho * (plan->shape.wo + halo_w);
    const int halo_k_iters = s->kh * plan->c_blocks;
    int pair = 0;
    // (grouped layers keep their 64-column tiles: a strip and kw weight tiles of that width always fit)
    const int bn = mv > 0x7fffffffLL ? 0
                   : grouped         ? (s->kw <= 7 ? kGroupedBlockN : 0)
                                     : pick_block_n_halo(s->cout, mv, halo_k_iters, s->kw, (kBlockM + halo_w) * 128, &pair,
                                                         nullptr);
    if (bn != 0) {
      plan->im2col = kModeHalo;
      plan->m_virtual = static_cast<int>(mv);
      plan->strip_rows = kBlockM + halo_w;
      plan->k_iters = halo_k_iters;
      plan->block_n = bn;
      plan->cta_pair = pair;
    }
  }
  const bool halo = plan->im2col == kModeHalo;
  const bool small = !grouped && small_tiles(s->cout, plan->m_virtual, plan->k_iters, halo ? s->kw : 1, halo ? halo_w : 0,
                                             segment_shift_of(plan->shape, plan->im2col, plan->k_iters), &plan->block_n, &plan->cta_pair);
  if (small) plan->strip_rows = kSmallM + (halo ? halo_w : 0);

  CUtensorMap* ma = reinterpret_cast<CUtensorMap*>(plan->tma_a);
  CUtensorMap* mb = reinterpret_cast<CUtensorMap*>(plan->tma_b);
  CUresult r;
  if (pointwise) {
    // Plain row-major matrix [m, c] with row pitch c_stride.
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(s->c), static_cast<cuuint64_t>(plan->m)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(s->c_stride) * es};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kelems), static_cast<cuuint32_t>(small ? kSmallM : kBlockM)};
    const cuuint32_t estr[2] = {1, 1};
    r = api.tiled(ma, dtype, 2, const_cast<void*>(in), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  } else {
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(s->c), static_cast<cuuint64_t>(s->w),
                                static_cast<cuuint64_t>(s->h), static_cast<cuuint64_t>(s->n)};
    const cuuint64_t pix = static_cast<cuuint64_t>(s->c_stride) * es;
    const cuuint64_t strides[3] = {pix, pix * s->w, pix * s->w * s->h};
    // Window of base pixels (top-left filter corners): starts at -pad and ends
    // where the last tap still lies inside the padded image.
    const int lower[2] = {-s->pad_w, -s->pad_h};
    // Halo mode walks every position of the padded row (w + 2 * pad_w of them), not only the wo
    // positions a filter's left edge can take: the extra ones are the taps' halo.
    const int upper[2] = {halo ? s->pad_w : s->pad_w - (s->kw - 1) * s->dil_w, s->pad_h - (s->kh - 1) * s->dil_h};
    const cuuint32_t estr[4] = {1, static_cast<cuuint32_t>(s->stride_w), static_cast<cuuint32_t>(s->stride_h), 1};
    r = api.im2col(ma, dtype, 4, const_cast<void*>(in), dims, strides, lower, upper,
                   static_cast<cuuint32_t>(kelems), static_cast<cuuint32_t>(plan->strip_rows ? plan->strip_rows : kBlockM), estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS) clear_small_tensor_flag(ma, pix * s->w * s->h * s->n);
  }
  if (r != CUDA_SUCCESS) return -100 - static_cast<int>(r);
  {
    const cuuint64_t kp = static_cast<cuuint64_t>(s->kh) * s->kw * plan->c_blocks * kelems;
    const cuuint64_t dims[2] = {kp, static_cast<cuuint64_t>(s->cout)};
    const cuuint64_t strides[1] = {kp * es};
    // A CTA of a pair fetches half of the weight tile.
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kelems),
                               static_cast<cuuint32_t>(plan->cta_pair ? plan->block_n / 2 : plan->block_n)};
    const cuuint32_t estr[2] = {1, 1};
    r = api.tiled(mb, dtype, 2, const_cast<void*>(packed_w), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -200 - static_cast<int>(r);
  }
  return 0;
}

int launch_core(mcb200_conv_plan* plan, void* out, bool out_half, int out_ld, const mcb200_epilogue* ep, int* status,
                void* stream, int flags = 0, const mcb200_deconv_plan* phases = nullptr, const mcb200_conv_second* second = nullptr);

}  // namespace

extern "C" int mcb200_conv_tc_plan(const mcb200_conv_shape* s, const float* in, const float* packed_w,
                                   mcb200_conv_plan* plan) {
  return plan_core(s, in, packed_w, plan, false);
}

extern "C" int mcb200_conv_tc_plan_bf16(const mcb200_conv_shape* s, const uint16_t* in, const uint16_t* packed_w,
                                        mcb200_conv_plan* plan) {
  return plan_core(s, in, packed_w, plan, true);
}

extern "C" int mcb200_conv_tc_launch(mcb200_conv_plan* plan, float* out, int out_ld, const mcb200_epilogue* ep,
                                     int* status, void* stream) {
  if (plan && plan->operand_bf16) return -8;   // bfloat16 plans go through mcb200_conv_tc_launch_bf16
  return launch_core(plan, out, false, out_ld, ep, status, stream);
}

extern "C" int mcb200_conv_tc_launch_flags(mcb200_conv_plan* plan, void* out, int out_is_bf16, int out_ld,
                                           const mcb200_epilogue* ep, int flags, int* status, void* stream) {
  return launch_core(plan, out, out_is_bf16 != 0, out_ld, ep, status, stream, flags);
}

extern "C" int mcb200_conv_tc_launch_bf16(mcb200_conv_plan* plan, void* out, int out_is_bf16, int out_ld,
                                          const mcb200_epilogue* ep, int* status, void* stream) {
  return launch_core(plan, out, out_is_bf16 != 0, out_ld, ep, status, stream);
}

extern "C" int mcb200_conv_tc_launch_two(mcb200_conv_plan* plan, void* out, int out_is_bf16, int out_ld, const mcb200_epilogue* ep,
                                         const mcb200_conv_second* second, int flags, int* status, void* stream) {
  if (!second) return -1;
  return launch_core(plan, out, out_is_bf16 != 0, out_ld, ep, status, stream, flags, nullptr, second);
}

namespace {

int launch_core(mcb200_conv_plan* plan, void* out, bool out_half, int out_ld, const mcb200_epilogue* ep, int* status,
                void* stream, int flags, const mcb200_deconv_plan* phases, const mcb200_conv_second* second) {
  if (!plan || !out || out_ld < (second ? second->first_cout : plan->shape.cout)) return -1;
  const bool half = plan->operand_bf16 != 0;
  ConvTcArgs a;
  a.out = static_cast<float*>(out);
  a.out_half = out_half ? 1 : 0;
  a.out_ld = out_ld;
  a.m = plan->m;
  a.cout = plan->shape.cout;
  a.k_iters = plan->k_iters;
  a.c_blocks = plan->c_blocks;
  a.kw = plan->shape.kw;
  a.ho = plan->shape.ho;
  a.wo = plan->shape.wo;
  a.stride_h = plan->shape.stride_h;
  a.stride_w = plan->shape.stride_w;
  a.pad_h = plan->shape.pad_h;
  a.pad_w = plan->shape.pad_w;
  a.dil_h = plan->shape.dil_h;
  a.dil_w = plan->shape.dil_w;
  if (ep) {
    a.ep = *ep;
  } else {
    a.ep = mcb200_epilogue();
    a.ep.residual_coeff = 1.f;
  }
  if (a.ep.act == 2 && !a.ep.prelu) return -2;
  a.second_begin = 0x7fffffff;
  a.first_cout = a.cout;
  a.second_out = nullptr;
  a.second_ld = a.second_act = 0;
  if (second) {
    const int columns = a.cout - second->begin;
    if (second->begin % 32 != 0 || second->first_cout < 1 || second->first_cout > second->begin || columns < 1 || !second->out ||
        second->out_ld < columns || a.ep.residual || a.ep.act > 1 || a.ep.slope != 0.f || second->act < 0 || second->act > 1 ||
        plan->shape.group != 1 || plan->im2col == kModeRows || phases)
      return -9;
    a.second_begin = second->begin;
    a.first_cout = second->first_cout;
    a.second_out = static_cast<float*>(second->out);
    a.second_ld = second->out_ld;
    a.second_act = second->act;
  }
  a.status = status;
  // Wide accesses of the epilogue: pairs of fp32 columns, eight bfloat16 columns of the output, pairs of the residual.
  const int wide = out_half ? 8 : 2;
  auto wide_ok = [&](const void* to, int ld, int columns) {
    return ld % wide == 0 && columns % wide == 0 && (reinterpret_cast<uintptr_t>(to) & (out_half ? 15 : 7)) == 0;
  };
  const bool out_ok = wide_ok(out, out_ld, a.first_cout) &&
                      (!second || wide_ok(second->out, second->out_ld, a.cout - second->begin));
  const bool res_ok = !a.ep.residual || (a.ep.residual_ld % 2 == 0 && a.cout % 2 == 0 &&
                                         (reinterpret_cast<uintptr_t>(a.ep.residual) & (half ? 3 : 7)) == 0);
  a.vec_store = out_ok && res_ok ? 1 : 0;
  a.l2_prefetch = 0;
  a.wait_limit = g_wait_limit_cycles;
  a.constants_settled = (flags & MCB200_CONV_CONSTANTS_SETTLED) ? 1 : 0;
  a.drop_last_weight_load = conv_take_drop_hook();
  a.group_cout = plan->shape.group > 1 ? plan->shape.cout / plan->shape.group : 0;
  a.group_cin = plan->shape.group > 1 ? plan->shape.c / plan->shape.group : 0;
  a.wp = plan->shape.wo;
  a.stage_bytes = a.stage_b_offset = a.resident_b_bytes = 0;
  if (plan->im2col == kModeHalo) {
    a.m = plan->m_virtual;
    a.wp = plan->m_virtual / (plan->shape.n * plan->shape.ho);
  }
  a.phase_tiles = 0;
  if (phases) {
    a.phase_tiles = (a.cout + plan->block_n - 1) / plan->block_n;
    a.phase_stride_h = phases->stride_h;
    a.phase_stride_w = phases->stride_w;
    for (int i = 0; i < kMaxPhase; ++i) {
      a.phase_off_h[i] = phases->off_h[i];
      a.phase_off_w[i] = phases->off_w[i];
    }
    a.out_h = phases->out_h;
    a.out_w = phases->out_w;
    a.ho = phases->grid_h;
    a.wo = phases->grid_w;
  }
  const bool small = m_tile_of(*plan) == kSmallM;
  a.segment_shift = plan_segment_shift(*plan);
  const bool split = split_launch(*plan, a.segment_shift);
  // Tile maps of output and residual: rows of 16-byte cells, one box per sub-tile.
  auto cells_ok = [&](const void* to, int ld) { return ld % (out_half ? 8 : 4) == 0 && (reinterpret_cast<uintptr_t>(to) & 15) == 0; };
  const bool tma_ok = cells_ok(out, out_ld) && (!second || cells_ok(second->out, second->out_ld)) &&
                      (!a.ep.residual || (a.ep.residual_ld % (half ? 8 : 4) == 0 && a.ep.residual_ld >= a.cout &&
                                          (reinterpret_cast<uintptr_t>(a.ep.residual) & 15) == 0));
  const bool cut_or_rows = plan->im2col == kModeMatrix || plan->im2col == kModeIm2col || plan->im2col == kModeRows;
  const bool staged = cut_or_rows && !small && tma_ok && a.segment_shift == 0 && staged_epilogue(plan, a.ep.residual != nullptr);
  if (staged) {
    const bool rows = plan->im2col == kModeRows;
    const long long per_group = rows ? plan->shape.wo : plan->m;
    const long long groups = rows ? static_cast<long long>(plan->shape.n) * plan->shape.ho : 1;
    // The maps are kept for the next launch to the same places, of as many layers.
    const int kind = a.out_half | (second ? 2 * a.first_cout : 0);
    const bool new_out = plan->out_ptr != out || plan->out_ld != out_ld || plan->out_bf16 != kind;
    if (new_out) {
      if (encode_tile_map(reinterpret_cast<CUtensorMap*>(plan->tma_out), out, out_half, a.first_cout, out_ld,
                          per_group, groups) != CUDA_SUCCESS)
        return -4;
      plan->out_ptr = static_cast<const float*>(out);
      plan->out_ld = out_ld;
      plan->out_bf16 = kind;
    }
    if (second && (plan->res_ptr != second->out || plan->res_ld != second->out_ld || new_out)) {
      if (encode_tile_map(reinterpret_cast<CUtensorMap*>(plan->tma_res), second->out, out_half, a.cout - second->begin,
                          second->out_ld, per_group, groups) != CUDA_SUCCESS)
        return -5;
      plan->res_ptr = static_cast<const float*>(second->out);
      plan->res_ld = second->out_ld;
    }
    if (a.ep.residual && (plan->res_ptr != a.ep.residual || plan->res_ld != a.ep.residual_ld || new_out)) {
      if (encode_tile_map(reinterpret_cast<CUtensorMap*>(plan->tma_res), a.ep.residual, half, plan->shape.cout,
                          a.ep.residual_ld, per_group, groups) != CUDA_SUCCESS)
        return -5;
      plan->res_ptr = a.ep.residual;
      plan->res_ld = a.ep.residual_ld;
    }
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  a.tile_rows = plan->im2col == kModeRows ? (plan->shape.wo < kBlockM ? plan->shape.wo : kBlockM) : small ? kSmallM : kBlockM;
  a.row_segments = plan->im2col == kModeRows ? (plan->shape.wo + a.tile_rows - 1) / a.tile_rows : 1;
  a.a_bytes = (plan->im2col == kModeHalo ? plan->strip_rows : a.tile_rows) * kBlockK * 4;
  cudaError_t e = cudaErrorInvalidValue;
  const int mode = plan->im2col;
#define MCB200_OUT_ONE(BN, MODE, PAIR, HALF)                                                       \
  (staged ? launch_variant<BN, MODE, PAIR, HALF, kOutStaged>(plan, a, st) : launch_variant<BN, MODE, PAIR, HALF>(plan, a, st))
#define MCB200_OUT(BN, MODE, PAIR, HALF)                                                           \
  (staged && second ? launch_variant<BN, MODE, PAIR, HALF, kOutStagedTwo>(plan, a, st) : MCB200_OUT_ONE(BN, MODE, PAIR, HALF))
#define MCB200_DISPATCH(BN)                                                                        \
  e = mode == kModeRows     ? MCB200_OUT_ONE(BN, kModeRows, false, false)                          \
      : mode == kModeIm2col ? MCB200_OUT(BN, kModeIm2col, false, false)                            \
      : mode == kModeHalo   ? launch_variant<BN, kModeHalo, false, false>(plan, a, st)             \
      : mode == kModePhase  ? launch_variant<BN, kModePhase, false, false>(plan, a, st)            \
                            : MCB200_OUT(BN, kModeMatrix, false, false)
#define MCB200_DISPATCH_PAIR(BN)                                                                   \
  e = mode == kModeIm2col ? MCB200_OUT(BN, kModeIm2col, true, false)                               \
      : mode == kModeHalo ? launch_variant<BN, kModeHalo, true, false>(plan, a, st)                \
                          : MCB200_OUT(BN, kModeMatrix, true, false)
#define MCB200_DISPATCH_NARROW(HALF)                                                               \
  e = mode == kModeIm2col   ? launch_variant<32, kModeIm2col, false, HALF>(plan, a, st)            \
      : mode == kModeHalo   ? launch_variant<32, kModeHalo, false, HALF>(plan, a, st)              \
      : mode == kModeMatrix ? launch_variant<32, kModeMatrix, false, HALF>(plan, a, st)            \
                            : cudaErrorInvalidValue
#define MCB200_DISPATCH_HALF(BN, PAIR)                                                             \
  e = mode == kModeIm2col ? MCB200_OUT(BN, kModeIm2col, PAIR, true)                                \
      : mode == kModeHalo ? launch_variant<BN, kModeHalo, PAIR, true>(plan, a, st)                 \
                          : MCB200_OUT(BN, kModeMatrix, PAIR, true)
#define MCB200_DISPATCH_SPLIT(BN, HALF)                                                            \
  e = mode == kModeIm2col ? launch_variant<BN, kModeIm2col, false, HALF, kOutSplit>(plan, a, st)   \
      : mode == kModeHalo ? launch_variant<BN, kModeHalo, false, HALF, kOutSplit>(plan, a, st)     \
                          : launch_variant<BN, kModeMatrix, false, HALF, kOutSplit>(plan, a, st)
  if (split) {
    switch (plan->block_n * 2 + (half ? 1 : 0)) {
      case 64: MCB200_DISPATCH_SPLIT(32, false); break;
      case 65: MCB200_DISPATCH_SPLIT(32, true); break;
      case 128: MCB200_DISPATCH_SPLIT(64, false); break;
      case 129: MCB200_DISPATCH_SPLIT(64, true); break;
      case 256: MCB200_DISPATCH_SPLIT(128, false); break;
      case 257: MCB200_DISPATCH_SPLIT(128, true); break;
      default: return -3;
    }
    return static_cast<int>(e);
  }
  if (half) {
    if (mode == kModeRows) return -3;
    if (plan->cta_pair) {
      switch (plan->block_n) {
        case 128: MCB200_DISPATCH_HALF(128, true); break;
        case 256: MCB200_DISPATCH_HALF(256, true); break;
        default: return -3;
      }
    } else {
      switch (plan->block_n) {
        case 32: MCB200_DISPATCH_NARROW(true); break;
        case 64: MCB200_DISPATCH_HALF(64, false); break;
        case 128: MCB200_DISPATCH_HALF(128, false); break;
        case 256: MCB200_DISPATCH_HALF(256, false); break;
        default: return -3;
      }
    }
    return static_cast<int>(e);
  }
  if (plan->cta_pair) {
    if (mode == kModeRows) return -3;
    switch (plan->block_n) {
      case 128: MCB200_DISPATCH_PAIR(128); break;
      case 256: MCB200_DISPATCH_PAIR(256); break;
      default: return -3;
    }
    return static_cast<int>(e);
  }
  switch (plan->block_n) {
    case 32: MCB200_DISPATCH_NARROW(false); break;
    case 64: MCB200_DISPATCH(64); break;
    case 128: MCB200_DISPATCH(128); break;
    case 256: MCB200_DISPATCH(256); break;
    default: return -3;
  }
#undef MCB200_DISPATCH_NARROW
#undef MCB200_DISPATCH_HALF
#undef MCB200_DISPATCH_PAIR
#undef MCB200_DISPATCH
#undef MCB200_OUT
#undef MCB200_OUT_ONE
#undef MCB200_DISPATCH_SPLIT
  return static_cast<int>(e);
}

}  // namespace

// ------------------------------------------------------------------ phase mode (deconvolution)

namespace mcb200 {
namespace {

// Geometry of one axis: the filter window of phase f covers the input positions
// i + first[f] .. i + first[f] + taps - 1 for grid position i.
struct PhaseAxis {
  int taps, grid, lowest;      // lowest = min over the phases of `first`
  int first[kMaxPhase];
};

bool phase_axis(int k, int stride, int pad, int out, PhaseAxis* a) {
  if (stride < 1 || stride > kMaxPhase || out < 1) return false;
  a->taps = (k + stride - 1) / stride;
  a->grid = (out + stride - 1) / stride;
  for (int f = 0; f < stride; ++f) {
    // tap r reaches output i * stride + f from input i + (f + pad - r) / stride
    const int last = (f + pad - (f + pad) % stride) / stride;
    a->first[f] = last - (a->taps - 1);
    a->lowest = f == 0 || a->first[f] < a->lowest ? a->first[f] : a->lowest;
  }
  return true;
}

// A single input pixel reaches every output pixel through exactly one tap: the layer is then one
// phase per tap, whatever its stride.
void phase_strides(const mcb200_conv_shape& d, int* sh, int* sw) {
  const bool pixel = d.h == 1 && d.w == 1 && d.pad_h == 0 && d.pad_w == 0;
  *sh = pixel ? d.kh : d.stride_h;
  *sw = pixel ? d.kw : d.stride_w;
}

struct PhaseTable {
  int first_h[kMaxPhase], first_w[kMaxPhase];
  int stride_h, stride_w, pad_h, pad_w, kh, kw, taps_h, taps_w;
};

// [c_in, c_out, kh, kw] -> [phase][c_out][taps][c_pad], zero where a window reaches past the filter.
__global__ void pack_phase_weights_kernel(const float* __restrict__ w, float* __restrict__ packed, int c, int cout, int c_pad,
                                          PhaseTable p) {
  const int taps = p.taps_h * p.taps_w;
  const size_t total = static_cast<size_t>(p.stride_h) * p.stride_w * cout * taps * c_pad;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int cc = static_cast<int>(i % c_pad);
    const int tap = static_cast<int>((i / c_pad) % taps);
    const size_t row = i / (static_cast<size_t>(c_pad) * taps);
    const int co = static_cast<int>(row % cout), phase = static_cast<int>(row / cout);
    const int py = phase / p.stride_w, px = phase % p.stride_w;
    const int r = py + p.pad_h - p.stride_h * (p.first_h[py] + tap / p.taps_w);
    const int q = px + p.pad_w - p.stride_w * (p.first_w[px] + tap % p.taps_w);
    float v = 0.f;
    if (cc < c && r >= 0 && r < p.kh && q >= 0 && q < p.kw)
      v = round_to_tf32(w[((static_cast<size_t>(cc) * cout + co) * p.kh + r) * p.kw + q]);
    packed[i] = v;
  }
}

bool phase_geometry(const mcb200_conv_shape* deconv, mcb200_conv_shape* d, PhaseAxis* y, PhaseAxis* x, int* sh, int* sw) {
  if (!deconv) return false;
  *d = *deconv;
  if (mcb200_deconv_out_shape(d) != 0) return false;
  if (d->group != 1 || d->dil_h != 1 || d->dil_w != 1 || d->c_stride < d->c || (d->c_stride & 3) != 0) return false;
  phase_strides(*d, sh, sw);
  if (!phase_axis(d->kh, *sh, d->pad_h, d->ho, y) || !phase_axis(d->kw, *sw, d->pad_w, d->wo, x)) return false;
  // limits of the im2col tensor map: 8-bit signed box corners
  const int upper_h = y->grid - d->h + y->lowest, upper_w = x->grid - d->w + x->lowest;
  return y->lowest >= -128 && x->lowest >= -128 && upper_h >= -128 && upper_h <= 127 && upper_w >= -128 && upper_w <= 127 &&
         static_cast<long long>(d->n) * y->grid * x->grid <= 0x7fffffffLL;
}

}  // namespace
}  // namespace mcb200

extern "C" size_t mcb200_deconv_tc_packed_weight_count(const mcb200_conv_shape* deconv) {
  mcb200_conv_shape d;
  PhaseAxis y, x;
  int sh, sw;
  if (!phase_geometry(deconv, &d, &y, &x, &sh, &sw)) return 0;
  return static_cast<size_t>(sh) * sw * d.cout * y.taps * x.taps * ((d.c + kBlockK - 1) / kBlockK * kBlockK);
}

extern "C" int mcb200_deconv_tc_pack_weights(const mcb200_conv_shape* deconv, const float* w_iohw, float* packed, void* stream) {
  mcb200_conv_shape d;
  PhaseAxis y, x;
  int sh, sw;
  if (!w_iohw || !packed || !phase_geometry(deconv, &d, &y, &x, &sh, &sw)) return -1;
  PhaseTable t = {};
  for (int f = 0; f < kMaxPhase; ++f) {
    t.first_h[f] = y.first[f];
    t.first_w[f] = x.first[f];
  }
  t.stride_h = sh;
  t.stride_w = sw;
  t.pad_h = d.pad_h;
  t.pad_w = d.pad_w;
  t.kh = d.kh;
  t.kw = d.kw;
  t.taps_h = y.taps;
  t.taps_w = x.taps;
  const size_t total = mcb200_deconv_tc_packed_weight_count(deconv);
  const size_t blocks = (total + 255) / 256;
  pack_phase_weights_kernel<<<static_cast<int>(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w_iohw, packed, d.c, d.cout, (d.c + kBlockK - 1) / kBlockK * kBlockK, t);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

namespace mcb200 {
namespace {

// [c_in, c_out, kh, kw] -> [phase][c_out][c_in][window_h][window_w] over the union of the phases'
// windows, zero where a phase's filter does not reach.
__global__ void window_weights_kernel(const float* __restrict__ w, float* __restrict__ out, int c, int cout, int win_h, int win_w,
                                      int lowest_h, int lowest_w, PhaseTable p) {
  const size_t total = static_cast<size_t>(p.stride_h) * p.stride_w * cout * c * win_h * win_w;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    size_t t = i;
    const int tx = static_cast<int>(t % win_w);
    t /= win_w;
    const int ty = static_cast<int>(t % win_h);
    t /= win_h;
    const int cc = static_cast<int>(t % c);
    t /= c;
    const int co = static_cast<int>(t % cout), phase = static_cast<int>(t / cout);
    const int r = phase / p.stride_w + p.pad_h - p.stride_h * (lowest_h + ty);
    const int q = phase % p.stride_w + p.pad_w - p.stride_w * (lowest_w + tx);
    out[i] = r >= 0 && r < p.kh && q >= 0 && q < p.kw ? w[((static_cast<size_t>(cc) * cout + co) * p.kh + r) * p.kw + q] : 0.f;
  }
}

// The window of an axis and whether a stride-1 convolution padded alike on both ends yields the grid.
bool window_of(const PhaseAxis& a, int stride, int size, int* window) {
  int highest = a.first[0];
  for (int f = 1; f < stride; ++f) highest = a.first[f] > highest ? a.first[f] : highest;
  *window = highest + a.taps - a.lowest;
  return a.lowest <= 0 && size - 2 * a.lowest - *window + 1 == a.grid;
}

}  // namespace
}  // namespace mcb200

extern "C" int mcb200_deconv_as_window_conv(const mcb200_conv_shape* deconv, mcb200_conv_shape* conv) {
  mcb200_conv_shape d;
  PhaseAxis y, x;
  int sh, sw, win_h, win_w;
  if (!conv || !phase_geometry(deconv, &d, &y, &x, &sh, &sw)) return -1;
  if (!window_of(y, sh, d.h, &win_h) || !window_of(x, sw, d.w, &win_w)) return -2;
  *conv = d;
  conv->cout = d.cout * sh * sw;
  conv->kh = win_h;
  conv->kw = win_w;
  conv->pad_h = -y.lowest;
  conv->pad_w = -x.lowest;
  conv->stride_h = conv->stride_w = 1;
  return mcb200_conv_out_shape(conv);
}

extern "C" int mcb200_deconv_window_weights(const mcb200_conv_shape* deconv, const float* w_iohw, float* w_oihw, void* stream) {
  mcb200_conv_shape d, conv;
  PhaseAxis y, x;
  int sh, sw;
  if (!w_iohw || !w_oihw || mcb200_deconv_as_window_conv(deconv, &conv) != 0 || !phase_geometry(deconv, &d, &y, &x, &sh, &sw)) return -1;
  PhaseTable t = {};
  t.stride_h = sh;
  t.stride_w = sw;
  t.pad_h = d.pad_h;
  t.pad_w = d.pad_w;
  t.kh = d.kh;
  t.kw = d.kw;
  const size_t total = static_cast<size_t>(conv.cout) * d.c * conv.kh * conv.kw;
  const size_t blocks = (total + 255) / 256;
  window_weights_kernel<<<static_cast<int>(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w_iohw, w_oihw, d.c, d.cout, conv.kh, conv.kw, y.lowest, x.lowest, t);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_deconv_tc_plan(const mcb200_conv_shape* deconv, const float* in, const float* packed_w,
                                     mcb200_deconv_plan* plan) {
  mcb200_conv_shape d;
  PhaseAxis y, x;
  int sh, sw;
  if (!in || !packed_w || !plan) return -1;
  if (!phase_geometry(deconv, &d, &y, &x, &sh, &sw)) return -2;
  if ((reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(packed_w) & 15)) return -3;
  const DriverApi& api = driver_api();
  if (!api.ok) return -5;
  mcb200_conv_plan& conv = plan->conv;
  conv.shape = d;
  conv.shape.kh = y.taps;
  conv.shape.kw = x.taps;
  conv.shape.stride_h = conv.shape.stride_w = 1;
  conv.shape.pad_h = -y.lowest;
  conv.shape.pad_w = -x.lowest;
  conv.out_ptr = nullptr;
  conv.res_ptr = nullptr;
  conv.out_ld = conv.res_ld = conv.cta_pair = 0;
  conv.operand_bf16 = conv.out_bf16 = 0;
  conv.m = d.n * y.grid * x.grid;
  conv.m_virtual = conv.m;
  conv.strip_rows = 0;
  conv.c_blocks = (d.c + kBlockK - 1) / kBlockK;
  conv.k_iters = y.taps * x.taps * conv.c_blocks;
  conv.im2col = kModePhase;
  plan->stride_h = sh;
  plan->stride_w = sw;
  plan->grid_h = y.grid;
  plan->grid_w = x.grid;
  plan->out_h = d.ho;
  plan->out_w = d.wo;
  for (int f = 0; f < kMaxPhase; ++f) {
    plan->off_h[f] = static_cast<unsigned char>(f < sh ? y.first[f] - y.lowest : 0);
    plan->off_w[f] = static_cast<unsigned char>(f < sw ? x.first[f] - x.lowest : 0);
  }
  // The phases multiply the tiles like so many more output pixels.
  conv.block_n = pick_block_n(d.cout, static_cast<long long>(conv.m) * sh * sw, conv.k_iters, 256);
  CUtensorMap* ma = reinterpret_cast<CUtensorMap*>(conv.tma_a);
  CUtensorMap* mb = reinterpret_cast<CUtensorMap*>(conv.tma_b);
  const cuuint64_t pix = static_cast<cuuint64_t>(d.c_stride) * 4;
  {
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(d.c), static_cast<cuuint64_t>(d.w), static_cast<cuuint64_t>(d.h),
                                static_cast<cuuint64_t>(d.n)};
    const cuuint64_t strides[3] = {pix, pix * d.w, pix * d.w * d.h};
    // Base pixels: as many positions per row and image as the grid has, from the lowest window start on.
    const int lower[2] = {x.lowest, y.lowest};
    const int upper[2] = {x.grid - d.w + x.lowest, y.grid - d.h + y.lowest};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = api.im2col(ma, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(in), dims, strides, lower, upper, kBlockK,
                            kBlockM, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -100 - static_cast<int>(r);
    clear_small_tensor_flag(ma, pix * d.w * d.h * d.n);
  }
  {
    const cuuint64_t kp = static_cast<cuuint64_t>(conv.k_iters) * kBlockK;
    const cuuint64_t dims[2] = {kp, static_cast<cuuint64_t>(d.cout) * sh * sw};
    const cuuint64_t strides[1] = {kp * 4};
    const cuuint32_t box[2] = {kBlockK, static_cast<cuuint32_t>(conv.block_n)};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = api.tiled(mb, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(packed_w), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -200 - static_cast<int>(r);
  }
  return 0;
}

extern "C" int mcb200_deconv_tc_launch(mcb200_deconv_plan* plan, float* out, int out_ld, const mcb200_epilogue* ep, int flags,
                                       int* status, void* stream) {
  if (!plan || plan->conv.im2col != kModePhase || (ep && ep->residual)) return -1;
  return launch_core(&plan->conv, out, false, out_ld, ep, status, stream, flags, plan);
}

// ------------------------------------------------------------------ row mode (few input channels)

namespace mcb200 {
namespace {

__global__ void pack_rows_weights_kernel(const float* __restrict__ w, float* __restrict__ packed, int cout, int c,
                                         int kh, int kw) {
  const int total = cout * kh * kBlockK;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int e = i % kBlockK;          // 8 pixels x 4 channels of one filter row
    const int r = (i / kBlockK) % kh;
    const int co = i / (kBlockK * kh);
    const int sx = e >> 2, ch = e & 3;
    float v = 0.f;
    if (sx < kw && ch < c) v = round_to_tf32(w[((static_cast<size_t>(co) * c + ch) * kh + r) * kw + sx]);
    packed[i] = v;
  }
}

// (N, C<=4, H, W) -> zero-bordered channels-last copy with 4 floats per pixel.
__global__ void pad_nhwc4_kernel(const float* __restrict__ src, float4* __restrict__ dst, int n, int c, int h, int w,
                                 int pad_h, int pad_w, int hp, int wp) {
  grid_launch_dependents();   // the convolution behind this copy may set itself up meanwhile
  // (A form with one block row per padded image row and no index divisions was measured: 33.8 us
  // against 24.7 us for 64 x 3 x 224 x 224: many small blocks with three loads per thread.)
  const long long total = static_cast<long long>(n) * hp * wp;
  const size_t plane = static_cast<size_t>(h) * w;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int xp = static_cast<int>(i % wp);
    const int yp = static_cast<int>((i / wp) % hp);
    const int img = static_cast<int>(i / (static_cast<long long>(wp) * hp));
    const int x = xp - pad_w, y = yp - pad_h;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (x >= 0 && x < w && y >= 0 && y < h) {
      const float* s = src + static_cast<size_t>(img) * c * plane + static_cast<size_t>(y) * w + x;
      v.x = s[0];
      if (c > 1) v.y = s[plane];
      if (c > 2) v.z = s[2 * plane];
      if (c > 3) v.w = s[3 * plane];
    }
    dst[i] = v;
  }
}

}  // namespace
}  // namespace mcb200

extern "C" int mcb200_conv_rows_supported(const mcb200_conv_shape* s) {
  if (!s || s->group != 1 || s->c < 1 || s->c > 4 || s->kw > 8 || s->dil_w != 1) return 0;
  mcb200_conv_shape t = *s;
  if (mcb200_conv_out_shape(&t) != 0) return 0;
  return t.wo >= 1;
}

extern "C" int mcb200_conv_rows_padded_dims(const mcb200_conv_shape* s, int* hp, int* wp) {
  if (!mcb200_conv_rows_supported(s) || !hp || !wp) return -1;
  mcb200_conv_shape t = *s;
  mcb200_conv_out_shape(&t);
  *hp = t.h + 2 * t.pad_h;
  const int reach = (t.wo - 1) * t.stride_w + 8;   // the last tile row reads 8 pixels
  *wp = t.w + 2 * t.pad_w > reach ? t.w + 2 * t.pad_w : reach;
  return 0;
}

extern "C" size_t mcb200_conv_rows_packed_weight_count(const mcb200_conv_shape* s) {
  return static_cast<size_t>(s->cout) * s->kh * kBlockK;
}

extern "C" int mcb200_conv_rows_pack_weights(const mcb200_conv_shape* s, const float* w_oihw, float* packed,
                                             void* stream) {
  if (!mcb200_conv_rows_supported(s) || !w_oihw || !packed) return -1;
  const int total = s->cout * s->kh * kBlockK;
  pack_rows_weights_kernel<<<(total + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(w_oihw, packed, s->cout,
                                                                                              s->c, s->kh, s->kw);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_conv_rows_pad_input(const mcb200_conv_shape* s, const float* src_nchw, float* padded,
                                          void* stream) {
  int hp = 0, wp = 0;
  if (mcb200_conv_rows_padded_dims(s, &hp, &wp) != 0 || !src_nchw || !padded) return -1;
  if (reinterpret_cast<uintptr_t>(padded) & 15) return -2;
  const long long total = static_cast<long long>(s->n) * hp * wp;
  if (total == 0) return 0;
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  pad_nhwc4_kernel<<<static_cast<int>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      src_nchw, reinterpret_cast<float4*>(padded), s->n, s->c, s->h, s->w, s->pad_h, s->pad_w, hp, wp);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

extern "C" int mcb200_conv_rows_plan(const mcb200_conv_shape* s, const float* padded_in, const float* packed_w,
                                     mcb200_conv_plan* plan) {
  if (!padded_in || !packed_w || !plan) return -1;
  int hp = 0, wp = 0;
  if (mcb200_conv_rows_padded_dims(s, &hp, &wp) != 0) return -2;
  if ((reinterpret_cast<uintptr_t>(padded_in) & 15) || (reinterpret_cast<uintptr_t>(packed_w) & 15)) return -3;
  const DriverApi& api = driver_api();
  if (!api.ok) return -5;
  plan->shape = *s;
  plan->shape.c_stride = 4;
  plan->out_ptr = nullptr;
  plan->res_ptr = nullptr;
  plan->out_ld = plan->res_ld = plan->cta_pair = 0;
  plan->operand_bf16 = plan->out_bf16 = 0;
  if (mcb200_conv_out_shape(&plan->shape) != 0) return -6;
  const long long m_ll = static_cast<long long>(s->n) * plan->shape.ho * plan->shape.wo;
  if (m_ll <= 0 || m_ll > 0x7fffffffLL) return -7;
  plan->m = static_cast<int>(m_ll);
  plan->m_virtual = plan->m;
  plan->strip_rows = 0;
  plan->c_blocks = 1;
  plan->k_iters = s->kh;
  plan->block_n = pick_block_n(s->cout, plan->m, plan->k_iters, 256);
  plan->im2col = kModeRows;
  // (Measured and dropped: a strip form that sorts the padded row into stride_w planes, loads a
  // filter row's pixels once (four to seven times fewer bytes out of L2) and lets the tensor core
  // read the windows through un-swizzled descriptors, rows 16 bytes apart.  Same values, but an
  // MMA with an un-swizzled operand occupied its issuing thread 76 cycles instead of 21, a 7 x 7
  // stride-2 first layer at batch 64 took 135 us instead of 106, and even the runtime switch
  // between the two forms cost the single-thread loops 100 cycles per filter row.)
  // Activation view: 32 floats (8 pixels x 4 channels) starting at padded pixel q * stride_w of padded row y.
  // Consecutive q overlap (the pitch of dimension 1 is stride_w pixels, less than the 8-pixel extent).
  CUtensorMap* ma = reinterpret_cast<CUtensorMap*>(plan->tma_a);
  const cuuint64_t dims[4] = {kBlockK, static_cast<cuuint64_t>(plan->shape.wo), static_cast<cuuint64_t>(hp),
                              static_cast<cuuint64_t>(s->n)};
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(s->stride_w) * 16, static_cast<cuuint64_t>(wp) * 16,
                                 static_cast<cuuint64_t>(wp) * 16 * hp};
  // One M tile = up to 128 output pixels of a row; wider rows are cut into segments.
  const cuuint32_t box[4] = {kBlockK, static_cast<cuuint32_t>(plan->shape.wo < kBlockM ? plan->shape.wo : kBlockM), 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = api.tiled(ma, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(padded_in), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return -100 - static_cast<int>(r);
  CUtensorMap* mb = reinterpret_cast<CUtensorMap*>(plan->tma_b);
  const cuuint64_t kp = static_cast<cuuint64_t>(plan->k_iters) * kBlockK;
  const cuuint64_t bdims[2] = {kp, static_cast<cuuint64_t>(s->cout)};
  const cuuint64_t bstrides[1] = {kp * 4};
  const cuuint32_t bbox[2] = {kBlockK, static_cast<cuuint32_t>(plan->block_n)};
  const cuuint32_t bestr[2] = {1, 1};
  r = api.tiled(mb, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(packed_w), bdims, bstrides, bbox, bestr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return -200 - static_cast<int>(r);
  return 0;
}

// With -DMCB200_CONV_TRACE: copies the cycle stamps of the last traced launches' CTA 0 (5 roles x
// 2048 slots, see MCB200_TRACE above) to `out` and clears the device array; returns the number
// of values per role, or 0 when the library was built without the trace.
extern "C" int mcb200_conv_trace_read(long long* out) {
#ifdef MCB200_CONV_TRACE
  if (!out) return -1;
  if (cudaDeviceSynchronize() != cudaSuccess) return -2;
  if (cudaMemcpyFromSymbol(out, mcb200::g_conv_trace, sizeof(long long) * mcb200::kTraceRoles * mcb200::kTraceSlots) !=
      cudaSuccess)
    return -3;
  static long long zeros[mcb200::kTraceRoles * mcb200::kTraceSlots];
  if (cudaMemcpyToSymbol(mcb200::g_conv_trace, zeros, sizeof(zeros)) != cudaSuccess) return -4;
  return mcb200::kTraceSlots;
#else
  (void)out;
  return 0;
#endif
}
