// Tensor-core W4A16 GEMM for sm_100a: out[M,N] = A[M,K] x dequant(W4[K,N]).
//
// Blackwell-native design: TMA-staged operands, in-kernel dequantization to fp16,
// tcgen05.mma with fp32 accumulators in tensor memory (TMEM).  The product is
// computed transposed ("swap-AB"): the 128 weight columns of a tile are the MMA's
// M side, up to 256 activation rows its N side, so one dequantized weight element
// feeds 256 multiply-adds and small M wastes no tensor work.
//
//   D^T[128 n x BM m] (TMEM, fp32)  +=  Wdq^T[128 n x 64 k] (TMEM, fp16)  x  A[BM m x 64 k]^T (smem)
//
// The dequantized weights never touch shared memory: the dequantizer threads write them
// straight into tensor memory (tcgen05.st) and the MMA takes its first operand from there.
// Measured with the operand staged in shared memory instead, the 16 KB written plus 16 KB
// re-read per step, on top of the TMA traffic, cost a third of the step time.
//
// Two kernels share this design.  gemm_tc_kernel (this file) gives every tile to one CTA, or its K range to a
// cluster of CTAs: M < 256, the larger skinny problems of gemm_tc_takes_skinny among them, and larger M with few
// tiles or short K (plan_tc).  gemm_tc_pair_kernel (blkq4_gemm_tc_pair.cuh; M >= 256) gives a 256 x 256 tile to a CTA pair.
//
// Persistent CTAs (one per SM) walk the tile list.  Warp roles of the one-CTA kernel, in the order of the warps (struct Shape:
// NG dequantizer groups, three or four):
//   0 to 3              epilogue: tcgen05.ld -> fp16 -> global, overlapped with the next tile
//                       through a second TMEM accumulator buffer where two fit
//   kFirstDeqWarp (4)   dequantizers, NG groups of four warps on steps in turn: thread = one
//                       weight column n of the tile (TMEM lane n), 64 k = 32 TMEM columns
//   kActProducerWarp    TMA producer of the activation tiles (128-byte swizzle); 4 + 4 NG
//   kWeightProducerWarp TMA producer of the packed int4 weight tiles
//   kMetaProducerWarp   TMA producer of their scales and zero points
//   kMmaWarp            MMA issuer (one elected thread), the last warp; owns the TMEM allocation
// A step is 64 k, or 128 k for tiles of up to 128 rows (struct Shape).
// Stages are handed over with mbarriers; every such wait, and every wait for another CTA's flag word, is bounded
// and, on expiry, sets an error word and drains the CTA instead of hanging the GPU.  The cluster barriers of
// a split have no limit of their own: every CTA of the cluster is resident and reaches them after bounded waits.
//
// The packed weight layout was designed for mma.sync register fragments (reference
// src/mickey/blk_q4/f16_quant_sm80.cuh:362-417); a 16-byte run of a packed column
// still holds 16 consecutive k of two columns n0, n0 + 8, so the threads of columns n0 and
// n0 + 8 read the same 64 bytes per step and each keeps its own nibbles.  Dequantization numerics are the
// reference kernel's (fp16(16+q) by bit trick, fma.rn.f16 with rn(scale*(-16-zp));
// src/mickey/cutlass_ext/q4gemm/warp/quantb_meta_mma_tensor_op_tile_iterator.h:69-104, :436-543).
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "blkq4_common.cuh"
#include "blkq4_tc.cuh"
#include "blkq4_tma.cuh"
#include "ms_blkq4gemm.h"

namespace blkq4 {

__device__ int g_gemm_tc_error = 0;  // 0 ok; otherwise (role << 8) | barrier id of the wait that gave up

namespace {

using namespace tc;
// Two rings.  The weight path (TMA -> shared memory -> dequantize -> tensor memory -> MMA) has a
// loop latency of several step times and small stages, so it is the deeper one; the activation path
// (TMA -> shared memory -> MMA) is short but its stages are up to 32 KB.
constexpr int kWarpsPerDeqGroup = 4;  // one warp per quarter of the TMEM lanes
constexpr int kNumEpiWarps = 4;

// Shape of the one-CTA kernel, by activation rows per tile.
//   MAXM    most activation rows of a tile: the pitch of the activation stages, so that the MMA thread's
//           operand addresses are constants
//   KSUB    64-k sub-steps per pipeline step: what the roles hand to one another at a time
//   RING    stages of the activations in shared memory and of dequantized weights in tensor memory (32 * KSUB
//           columns each): one ring, so that one barrier collects everything the MMAs of a step read
//   WS      shared-memory stages of the packed weights and meta
//   NG      dequantizer groups of four warps, on steps in turn
template <int MAXM_, int KSUB_, int RING_, int WS_, int NG_>
struct Shape {
  static constexpr int MAXM = MAXM_, KSUB = KSUB_, RING = RING_, WS = WS_, NG = NG_;
  static constexpr int kStepK = BLOCK_K * KSUB;
  static constexpr int kActSubBytes = MAXM * 128, kActBytes = kActSubBytes * KSUB;
  static constexpr int kDeqTmemCols = RING * KSUB * kDeqCols;
  static constexpr int kFirstDeqWarp = kNumEpiWarps;
  static constexpr int kActProducerWarp = kFirstDeqWarp + 4 * NG;
  static constexpr int kWeightProducerWarp = kActProducerWarp + 1;
  static constexpr int kMetaProducerWarp = kActProducerWarp + 2;
  static constexpr int kMmaWarp = kActProducerWarp + 3;
  static constexpr int kThreads = 32 * (kMmaWarp + 1);
};
// Up to 128 rows the math of a 64-k step is shorter than its hand-overs (three barriers, a commit, the polls
// of five roles: ~400 cycles with loads, conversion and MMAs all left out), so a step carries 128 k.  Measured on
// B200, 64-k against 128-k steps with three groups each: K = 8192, N = 28672, block 128: M = 64 54.6 vs 43.9 us,
// M = 17 50.2 vs 40.3, M = 128 67.2 vs 58.0; M = 100, 4096 -> 11008 20.5 vs 16.3; M = 32, 4096 x 4096 10.1 vs 9.5.
// Above 128 rows two 64-k steps of activations per stage leave three stages only (rowwise M = 333: 24.8 vs 27.4 us).
// Four groups where a CTA has many steps: up to 64 rows the dequantizers' instructions set the pace, and the scheduler has more
// to choose from; the fourth group's start-up and its share of the ring only pay off after some 16 steps.  Three / four, us, block
// 64 column-wise with zero points: K = 8192, N = 28672 (97 steps a CTA): M = 17 43.0 / 41.6, M = 64 46.7 / 45.7 (block 128,
// symmetric 45.7 / 45.1); 11008 x 4096 (22) M = 40 13.6 / 13.3; 4096 x 11008 (32) M = 64 14.4 / 14.0; 2048 x 22528 (19) M = 64
// 13.5 / 13.2; 1024 x 14336 (8) 6.4 / 6.4; 4096 x 4096 (8) 8.9 / 9.0.
using ShapeSmall = Shape<64, 2, 6, 10, 3>;  // two accumulators + six stages of 64 TMEM columns = 512
using ShapeSmallLong = Shape<64, 2, 6, 10, 4>;
constexpr int kLongSteps = 16;
using ShapeMid = Shape<128, 2, 4, 8, 3>;    // two accumulators + four stages = 512
using ShapeLarge = Shape<256, 1, 6, 6, 3>;
// Activation rows of a tile, a multiple of `unit`: as few tiles of up to 256 rows as there can be, all of one height.
// Measured on B200 against tiles of 256 and a remainder, whose MMAs multiply rows that are not there, us: M = 300, 4096 x 28672
// 85.3 / 75.1; M = 333, 1024 x 28672 36.4 / 32.3; M = 400, 8192 x 22528 137.2 / 128.5.
inline int tile_rows(int M, int unit) {
  const int tiles = (M + 255) / 256, rows = (M + tiles - 1) / tiles;
  return (rows + unit - 1) / unit * unit;
}
// k per pipeline step of the kernel that takes tiles of BM rows
inline int step_k(int BM) { return BM <= 64 ? ShapeSmall::kStepK : BM <= 128 ? ShapeMid::kStepK : ShapeLarge::kStepK; }
constexpr long long kWaitCycles = 4000000000ll;  // ~2 s: far beyond any legitimate wait

struct Params {
  int M, N, K, block;
  int block_shift;   // log2(block)
  int BM;            // activation rows per tile = UMMA N (multiple of 16, <= 256)
  int m_tiles, n_tiles;
  int has_zp;
  int meta_rows;     // rows of the scale / zero-point box per step
  int acc_bufs;      // TMEM accumulator buffers: 2 when 2*BM + the dequantized stages fit in 512 columns
  int a_col0;        // first TMEM column of the dequantized stages
  uint32_t tmem_cols;  // allocation: power of two >= acc_bufs*BM + kDeqStages*kDeqCols
  uint32_t meta_row_bytes_s, meta_row_bytes_z;  // bytes per box row
  __half* out;
  const __half* bias;  // fp16 [N] added to the fp16 result, or null
  // Work items.  A tile's K range may be cut in parts that different CTAs compute.
  //   balanced == 0: item = (tile, part), part < split covering k_per_item steps (the last one what is
  //     left).  split == 1: CTA b takes items b, b + grid, ...  split > 1: one item per CTA, the parts of a
  //     tile form a cluster and exchange their fp32 partial tiles through distributed shared memory.
  //   balanced == 1: the (tile, k step) sequence of the whole problem is cut in one contiguous range
  //     per CTA (range_bound), so that every SM gets the same number of steps whatever the tile
  //     count; a tile that straddles two ranges has its tail computed FIRST by the later CTA
  //     (partial tile, slot = that CTA) and its head LAST by the earlier CTA, which adds the partial.
  int split;
  int k_per_item;      // steps per work item
  int num_items;       // tiles * split
  int balanced;
  int k_steps;         // steps of a tile: K / 64, or / 128 rounded up for tiles of up to 128 rows
  int min_part;        // one-CTA kernel: range_bound's minimum in steps
  int total_steps;     // tiles * k_steps
  float* ws_partials;  // balanced: [cta][BM][128] fp32
  int gather_bulk;         // pair kernel, gather mode: peer copies as cp.async.bulk of whole rows
  int n_fastest, n_pairs;  // pair kernel: tile order (0: the m tiles of a pair of weight columns run together; 1: the column pairs of an m tile)
  GemmGroup grp;       // kernels with G > 1: the weight matrices whose column tiles (pairs of tiles) follow one another
  GatherTable gt;      // pair kernel, gt.world > 0: the result goes to every rank's gathered buffer instead of `out`
  unsigned* ws_flags;  // balanced: [cta]: arrivals (self-resetting)
};

// Tensor maps of the G weight matrices of a launch.
template <int G>
struct WeightMaps {
  CUtensorMap pack[G], scale[G], zp[G];
};
// The matrix that column tile `t` of a launch belongs to, and what the epilogue needs of it.  A unit is one tile of
// 128 columns, or in the pair kernel two.
struct Columns {
  int matrix, unit;  // unit: of the matrix
  int N;
  __half* out;
  const __half* bias;
};
template <int G>
__device__ __forceinline__ Columns columns_of(const Params& p, int unit) {
  if constexpr (G == 1) {
    return Columns{0, unit, p.N, p.out, p.bias};
  } else {
    const int i = p.grp.of_tile(unit);
    return Columns{i, unit - p.grp.first_tile(i), p.grp.n[i], p.grp.out[i], p.grp.bias[i]};
  }
}

// ---- PTX wrappers ---------------------------------------------------------------------------

// Bounded wait on an mbarrier; see mbar_wait_bounded.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int who) {
  return mbar_wait_bounded(bar, parity, abort_flag, &g_gemm_tc_error, who, kWaitCycles);
}
// ---- work items -----------------------------------------------------------------------------

constexpr int kMinPartSteps = 4;  // a range boundary closer than this (in 64-k steps) to a tile boundary moves onto it
inline int min_part(int step_k) { return kMinPartSteps * BLOCK_K / step_k; }

// First step of CTA b's range in balanced mode (b == grid: the end of the last range).
__host__ __device__ inline int range_bound(int total_steps, int k_steps, int grid, int b, int min_part = kMinPartSteps) {
  int x = (int)((long long)b * total_steps / grid);
  const int r = x % k_steps;
  if (r < min_part) x -= r;
  else if (r > k_steps - min_part) x += k_steps - r;
  return x;
}

struct Item {
  int tile, ks0, count;
  int role;    // 0: whole tile; 1: writes its partial tile to `slot`; 2: adds the partial tile in `slot`; 3: part of a cluster's tile
  int slot;
};
struct ItemCursor {
  int pos, end;  // balanced: steps of the range still to do; otherwise: next item index, item count
};
__device__ __forceinline__ ItemCursor first_item(const Params& p) {
  ItemCursor c;
  if (p.balanced) {
    c.pos = range_bound(p.total_steps, p.k_steps, (int)gridDim.x, (int)blockIdx.x, p.min_part);
    c.end = range_bound(p.total_steps, p.k_steps, (int)gridDim.x, (int)blockIdx.x + 1, p.min_part);
  } else {
    c.pos = (int)blockIdx.x;
    c.end = p.num_items;
  }
  return c;
}
__device__ __forceinline__ bool next_item(const Params& p, ItemCursor& c, Item& it) {
  if (c.pos >= c.end) return false;
  if (p.balanced) {
    it.tile = c.pos / p.k_steps;
    it.ks0 = c.pos - it.tile * p.k_steps;
    it.count = min(p.k_steps - it.ks0, c.end - c.pos);
    // a range is longer than a tile, so a cut tile has exactly two parts: its tail opens the later
    // CTA's range, its head closes the earlier one's
    it.role = it.ks0 > 0 ? 1 : (it.count < p.k_steps ? 2 : 0);
    it.slot = (int)blockIdx.x + (it.role == 2 ? 1 : 0);
    c.pos += it.count;
  } else {
    const int split = p.split;
    it.tile = c.pos / split;
    const int part = c.pos - it.tile * split;
    it.ks0 = part * p.k_per_item;
    it.count = min(p.k_per_item, p.k_steps - it.ks0);
    it.role = split == 1 ? 0 : 3;
    it.slot = 0;
    c.pos += (int)gridDim.x;
  }
  return true;
}

// Owner of row group r4 of a split tile whose parts own `slice4` groups each: r4 / slice4 for r4 < 64 (a tile has at
// most 256 rows) without a division.
__host__ __device__ constexpr int slice_inverse(int slice4) { return 65536 / slice4 + 1; }
__host__ __device__ constexpr int slice_owner(int r4, int inv) { return (r4 * inv) >> 16; }
constexpr bool slice_owner_is_exact() {
  for (int s = 1; s <= 64; ++s)
    for (int r = 0; r < 64; ++r)
      if (slice_owner(r, slice_inverse(s)) != r / s) return false;
  return true;
}
static_assert(slice_owner_is_exact());

// ---- shared-memory plan ---------------------------------------------------------------------

struct SmemPlan {
  uint32_t act, pack, scale, zp, out, bars, total;
};
// rows: activation rows a stage has room for (a multiple of 8: 1024-aligned sub-tiles of 64 k)
__host__ __device__ constexpr SmemPlan make_plan(int rows, int kStages, int act_stages, int ksub, uint32_t out_bytes = 0) {
  SmemPlan p{};
  uint32_t o = 0;
  p.act = o;   o += act_stages * (uint32_t)(rows * 128 * ksub);
  p.pack = o;  o += kStages * kPackTileBytes * ksub;
  p.scale = o; o += kStages * kScaleTileBytes * ksub;
  p.zp = o;    o += kStages * kZpTileBytes * ksub;
  p.out = o;   o += out_bytes;  // output staging of the pair kernel's epilogue
  p.bars = o;  o += 512;
  p.total = o + 1024;  // slack to align the dynamic base to 1024
  return p;
}

// Barrier slots (8 bytes each) inside the barrier block.  A "step full" barrier collects what the MMAs of a step
// read: the bytes of its activation tile and the arrivals of its dequantizer warps.  An "MMA done" barrier frees the
// activation stage and the stage of dequantized weights of its step.
#define BLKQ4_TC_BARRIER_SLOTS(WS, RING)                                                                            \
  constexpr int kStages = (WS);                                                                                    \
  constexpr int BAR_FULL = 0;                            /* [kStages] packed weights + meta landed (-> dequantizers) */ \
  constexpr int BAR_PACK_FREE = BAR_FULL + kStages;      /* [kStages] packed weights / meta read (-> producer) */   \
  constexpr int BAR_STEP_FULL = BAR_PACK_FREE + kStages; /* [ring] operands of the step are there (-> MMA issuer) */ \
  constexpr int BAR_MMA_DONE = BAR_STEP_FULL + (RING);   /* [ring] MMAs of the step retired */                      \
  constexpr int BAR_ACC_FULL = BAR_MMA_DONE + (RING);    /* [2] accumulator complete */                             \
  constexpr int BAR_ACC_EMPTY = BAR_ACC_FULL + 2;        /* [2] accumulator drained by the epilogue */              \
  constexpr int BAR_COUNT = BAR_ACC_EMPTY + 2;                                                                      \
  static_assert(BAR_COUNT * 8 + 16 <= 512, "barrier block too small");

template <bool COLWISE, class S, int G>
__global__ void __launch_bounds__(S::kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_act, const __grid_constant__ WeightMaps<G> wm, const Params p) {
  constexpr int KSUB = S::KSUB, kRing = S::RING, kStepK = S::kStepK;
  constexpr int kStepCols = kDeqCols * KSUB, kStepPackBytes = kPackTileBytes * KSUB;
  constexpr int kStepScaleBytes = kScaleTileBytes * KSUB, kStepZpBytes = kZpTileBytes * KSUB;
  BLKQ4_TC_BARRIER_SLOTS(S::WS, kRing)
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  constexpr SmemPlan plan = make_plan(S::MAXM, kStages, kRing, KSUB);
  const uint32_t bars = base + plan.bars;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + plan.bars + BAR_COUNT * 8);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + plan.bars + BAR_COUNT * 8 + 8);
  auto bar = [&](int id) { return bars + 8u * (uint32_t)id; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem_cols = p.tmem_cols;
  // Programmatic dependent launch: the next kernel of the stream may start its own set-up as soon
  // as every CTA of this one is resident.  In this kernel only the roles that touch activations,
  // the output or the split-K workspace wait for the preceding kernel (griddepcontrol.wait; it
  // returns at once for a plain launch); barrier set-up, TMEM allocation, the weight copies and the
  // dequantization of the first stages run ahead of it.
  asm volatile("griddepcontrol.launch_dependents;");

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bar(BAR_FULL + i), 2);  // the packed-tile producer and the meta producer, each with its bytes
      mbar_init(bar(BAR_PACK_FREE + i), kWarpsPerDeqGroup);
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(bar(BAR_STEP_FULL + i), kWarpsPerDeqGroup + 1);  // the dequantizer warps; the activation producer, with its bytes
      mbar_init(bar(BAR_MMA_DONE + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(BAR_ACC_FULL + i), 1);
      mbar_init(bar(BAR_ACC_EMPTY + i), kNumEpiWarps);
    }
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == S::kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == S::kActProducerWarp) {
    // ========================= TMA producer: activations ========================
    // A stage is free once the MMAs of the step that used it last have retired.
    if (elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");  // activations belong to stream order
      const uint32_t tx = (uint32_t)(p.BM * 128 * KSUB);
      uint32_t s = 0, free_par = 1;  // (the first round finds fresh barriers: the phase before their first one is complete)
      ItemCursor cur = first_item(p);
      Item item;
      while (next_item(p, cur, item)) {
        const int m_tile = item.tile % p.m_tiles;
        for (int ks = item.ks0; ks < item.ks0 + item.count; ++ks) {
          if (!mbar_wait(bar(BAR_MMA_DONE + s), free_par, abort_flag, 0x100 | s)) goto act_producer_done;
          const uint32_t fb = bar(BAR_STEP_FULL + s);
          mbar_arrive_expect_tx(fb, tx);
#pragma unroll
          for (int u = 0; u < KSUB; ++u)  // past the end of K the copy fills zeros
            tma_load_2d(base + plan.act + s * S::kActBytes + u * S::kActSubBytes, &tm_act, ks * kStepK + u * BLOCK_K,
                        m_tile * p.BM, fb);
          if (++s == kRing) { s = 0; free_par ^= 1u; }
        }
      }
    act_producer_done:;
    }
  } else if (warp == S::kWeightProducerWarp || warp == S::kMetaProducerWarp) {
    // ============ TMA producers: packed weights (one warp), scales and zero points (another) ============
    // Two producer threads, each arriving on the stage's barrier with its own byte count: the stage wait,
    // the byte-count post and up to three copies of a step are a serial chain for one thread.
    if (elect_one()) {
      const bool meta = warp == S::kMetaProducerWarp;
      const uint32_t tx = meta ? (uint32_t)p.meta_rows * p.meta_row_bytes_s +
                                     (p.has_zp ? (uint32_t)p.meta_rows * p.meta_row_bytes_z : 0u)
                               : (uint32_t)kStepPackBytes;
      uint32_t it = 0;
      ItemCursor cur = first_item(p);
      Item item;
      while (next_item(p, cur, item)) {
        const Columns col = columns_of<G>(p, item.tile / p.m_tiles);
        const int n_tile = col.unit;
        for (int ks = item.ks0; ks < item.ks0 + item.count; ++ks, ++it) {
          const int s = it % kStages;
          if (it >= (uint32_t)kStages &&
              !mbar_wait(bar(BAR_PACK_FREE + s), ((it / kStages) - 1) & 1, abort_flag, (meta ? 0x120 : 0x110) | s))
            goto w_producer_done;
          const uint32_t fb = bar(BAR_FULL + s);
          mbar_arrive_expect_tx(fb, tx);
          const int k0 = ks * kStepK;
          if (!meta) {
            tma_load_2d(base + plan.pack + s * kStepPackBytes, &wm.pack[col.matrix], k0, n_tile * (TILE_N / 2), fb);
          } else if (COLWISE) {
            // meta row-major [K/block, N]: box = meta_rows x 128 columns
            const int mrow = k0 >> p.block_shift;
            tma_load_2d(base + plan.scale + s * kStepScaleBytes, &wm.scale[col.matrix], n_tile * TILE_N, mrow, fb);
            if (p.has_zp) tma_load_2d(base + plan.zp + s * kStepZpBytes, &wm.zp[col.matrix], n_tile * TILE_N, mrow, fb);
          } else {
            // meta column-major [K, N/block]: box = meta_rows (n blocks) x 64 k
            const int mrow = (n_tile * TILE_N) >> p.block_shift;
            tma_load_2d(base + plan.scale + s * kStepScaleBytes, &wm.scale[col.matrix], k0, mrow, fb);
            if (p.has_zp) tma_load_2d(base + plan.zp + s * kStepZpBytes, &wm.zp[col.matrix], k0, mrow, fb);
          }
        }
      }
    w_producer_done:;
    }
  } else if (warp == S::kMmaWarp) {
    // =============================== MMA issuer =================================
    // One thread drives the tensor pipe: eight 128 x BM x 16 MMAs of a 128-k step take 130 cycles at BM = 16, 260 at
    // 64.  The dequantizer warps of the thread's scheduler compete with it for issue slots, so what the step holds besides
    // its MMAs sets the pace up to 128 rows.  Hence: one barrier per step; the ring unrolled, so that operand
    // and barrier addresses are constants; the poll of step i + 1 (non-blocking) ahead of the MMAs of step i; the
    // bounded, instrumented wait only where a poll fails; the last warp of the CTA (the scheduler favours it).  Measured on
    // B200, the loop alone beside three warps of dependent FMAs per scheduler, cycles a step at N = 16: two barriers and
    // ring indices 321, one barrier 262, the ring unrolled 143, as the last warp 131.
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(TILE_N, p.BM);
      const uint32_t desc_hi = (uint32_t)(make_sw128_kmajor_desc(0) >> 32);
      const uint32_t desc_lo_flags = (uint32_t)(make_sw128_kmajor_desc(0) & 0xFFFFFFFFu);  // LBO field
      const uint32_t act_lo0 = desc_lo_flags | (((base + plan.act) >> 4) & 0x3FFFu);
      const uint32_t a_tmem0 = tmem_base + (uint32_t)p.a_col0;
      ItemCursor cur = first_item(p);
      Item item;
      uint32_t tcount = 0, ab = 0, par_acc = 0, par = 0;
      bool ready = false;
      if (!next_item(p, cur, item)) goto mma_done;
      {
      uint32_t left = (uint32_t)item.count, accumulate = 0, d_tmem = tmem_base;
      for (;; par ^= 1u) {
#pragma unroll
        for (int s = 0; s < kRing; ++s) {
          const uint32_t full = bar(BAR_STEP_FULL + s);
          if (!ready && !mbar_try_wait(full, par) && !mbar_wait(full, par, abort_flag, 0x220 | s)) goto mma_done;
          tc_fence_after();
          ready = s + 1 < kRing ? mbar_test_wait(full + 8u, par) : mbar_test_wait(bar(BAR_STEP_FULL), par ^ 1u);
          // 16 k = 8 TMEM columns of the weights, 32 bytes (2 descriptor units) of the activation row
#pragma unroll
          for (int u = 0; u < KSUB; ++u)
            umma_f16_ts_x4(d_tmem, a_tmem0 + s * kStepCols + u * kDeqCols,
                           act_lo0 + ((s * S::kActBytes + u * S::kActSubBytes) >> 4), desc_hi, idesc, u > 0 ? 1u : accumulate);
          umma_commit(bar(BAR_MMA_DONE + s));
          accumulate = 1;
          if (--left == 0) {
            umma_commit(bar(BAR_ACC_FULL + ab));
            if (!next_item(p, cur, item)) goto mma_done;
            left = (uint32_t)item.count;
            accumulate = 0;
            if (++ab == (uint32_t)p.acc_bufs) { ab = 0; par_acc ^= 1u; }
            if (++tcount >= (uint32_t)p.acc_bufs && !mbar_wait(bar(BAR_ACC_EMPTY + ab), par_acc ^ 1u, abort_flag, 0x200 | ab))
              goto mma_done;
            tc_fence_after();
            d_tmem = tmem_base + ab * (uint32_t)p.BM;
          }
        }
      }
      }
    mma_done:;
    }
  } else if (warp < kNumEpiWarps) {
    // =============================== epilogue ===================================
    // A warp reads the TMEM lanes of its quarter (warp id % 4): lane = weight column n of
    // the tile, TMEM column = activation row m.  For one m the 32 lanes hold 32
    // consecutive n, i.e. 64 contiguous bytes of the row-major output.
    const int quarter = warp & 3;
    uint32_t tcount = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // output and workspace belong to stream order
    const size_t tile_floats = (size_t)p.BM * TILE_N;
    ItemCursor cur = first_item(p);
    Item item;
    for (; next_item(p, cur, item); ++tcount) {
      const Columns col = columns_of<G>(p, item.tile / p.m_tiles);
      const int n_tile = col.unit, m_tile = item.tile % p.m_tiles;
      const int ab = tcount % p.acc_bufs;
      if (!mbar_wait(bar(BAR_ACC_FULL + ab), (tcount / p.acc_bufs) & 1, abort_flag, 0x300 | ab)) break;
      tc_fence_after();
      auto load_acc = [&](int c0, uint32_t (&r)[32]) {
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        tmem_ld_32x32b_x32(lane_base + (uint32_t)(ab * p.BM + c0), r);
        tmem_ld_wait();
      };
      const int n_l = quarter * 32 + lane;
      if (item.role == 3) break;  // this CTA's only item: the cluster adds its parts up after the role branches
      if (item.role == 1) {
        // ---- a part that hands over: fp32 partial tile [m][n] to the workspace: for a row m
        //      the 32 lanes of a warp write 128 contiguous bytes.  (One line per lane, [n][m] with
        //      16-byte accesses, was measured slower: 32 lines touched per instruction.)
        float* dst_ws = p.ws_partials + (size_t)item.slot * tile_floats + n_l;
        const int rows = min(p.BM, p.M - m_tile * p.BM);
        for (int c0 = 0; c0 < rows; c0 += 32) {
          uint32_t r[32];
          load_acc(c0, r);
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c0 + j < rows) dst_ws[(size_t)(c0 + j) * TILE_N] = __uint_as_float(r[j]);
        }
        tc_fence_before();
        __threadfence();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar(BAR_ACC_EMPTY + ab));
          atomicAdd(p.ws_flags + item.slot, 1u);
        }
        continue;
      }
      if (item.role == 2) {
        // ---- the part that finishes the tile: wait (bounded) for the other part's partial tile ----
        if (lane == 0) {
          const unsigned want = (unsigned)kNumEpiWarps;
          const long long t0 = clock64();
          while (*reinterpret_cast<volatile unsigned*>(p.ws_flags + item.slot) < want) {
            if (*abort_flag || clock64() - t0 > kWaitCycles) {
              *abort_flag = 1;
              atomicCAS(&g_gemm_tc_error, 0, 0x320 | quarter);
              break;
            }
          }
          __threadfence();
        }
        __syncwarp();
        if (*abort_flag) break;
      }
      const float* src_ws = p.ws_partials + (size_t)item.slot * tile_floats + n_l;
      const int n = n_tile * TILE_N + quarter * 32 + lane;
      const int m0 = m_tile * p.BM, m_end = min(p.M, m0 + p.BM);  // a chunk of 32 rows may reach into the next tile
      // Lanes pair up (n even / odd) so that every store carries two adjacent n (4 bytes per
      // lane, 128 contiguous bytes per warp): the even lane writes the even rows m of a
      // 32-row chunk, the odd lane the odd rows, each with its partner's value alongside.
      const int odd = lane & 1;
      const uint32_t pick = trade_selector(odd);
      const bool n_ok = (n | 1) < col.N;  // N is a multiple of 16: the pair is in or out together
      for (int c0 = 0; c0 < p.BM; c0 += 32) {
        if (m0 + c0 >= m_end) break;  // warp-uniform
        uint32_t r[32];
        load_acc(c0, r);
        if (item.role == 2) {
          const float* sq = src_ws + (size_t)c0 * TILE_N;
          float f[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = (m0 + c0 + j < m_end) ? __ldcg(sq + (size_t)j * TILE_N) : 0.0f;
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + f[j]);
        }
        int m = m0 + c0 + odd;
        __half* dst = col.out + (size_t)m * col.N + (n & ~1);
        // The bias is added to the ROUNDED result in fp16, which is what a separate
        // `output += bias` on the fp16 tensor computes.
        const bool add_bias = col.bias != nullptr && n_ok;
        const __half2 bias2 = add_bias ? *reinterpret_cast<const __half2*>(col.bias + (n & ~1)) : __half2();
        const size_t row_step = 2 * (size_t)col.N;
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const uint32_t traded = trade_rows(r[j], r[j + 1], pick);
          __half2 v = *reinterpret_cast<const __half2*>(&traded);
          if (add_bias) v = __hadd2(v, bias2);
          if (n_ok && m < m_end) *reinterpret_cast<__half2*>(dst) = v;
          dst += row_step;
          m += 2;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar(BAR_ACC_EMPTY + ab));
        // the warp that completes the tile's count puts the flag back to zero for the next launch
        if (item.role == 2 && atomicAdd(p.ws_flags + item.slot, 1u) == (unsigned)(2 * kNumEpiWarps - 1))
          p.ws_flags[item.slot] = 0u;
      }
    }
  } else {
    // =============================== dequantizers ===============================
    // The groups of four warps take steps in turn, so that a group has as many step times as there are
    // groups for the dependent chain wait -> load -> convert -> tcgen05.st -> arrive of one step.
    // A warp may only touch the TMEM lanes of its quarter (warp id % 4), and lane = row of the
    // MMA's first operand = weight column n of the tile: thread <-> n = 32 (warp % 4) + lane.
    // Column n lives in packed column np_l = 8 (n / 16) + n % 8 of the tile, in the "low"
    // nibble positions when n % 16 < 8 and 8 bits further up otherwise (the thread of n +- 8
    // reads the same bytes).  Per 64 k it reads the column's 64 bytes and writes 32 TMEM
    // columns: column j = fp16 pair k = (2j, 2j + 1).
    const int group = (warp - S::kFirstDeqWarp) / kWarpsPerDeqGroup;
    const int n_l = 32 * (warp & 3) + lane;
    const int np_l = 8 * (n_l >> 4) + (n_l & 7);
    const uint32_t rot_lo = (n_l & 8) ? 30u : 6u, rot_hi = (n_l & 8) ? 26u : 2u;
    const uint32_t tmem_row = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)p.a_col0;
    uint32_t total_its = 0;
    {
      ItemCursor cur = first_item(p);
      Item item;
      while (next_item(p, cur, item)) total_its += (uint32_t)item.count;
    }
    with_block_shift(p.block_shift, p.has_zp, [&](auto bsh, auto zp) {
    for (uint32_t it = group; it < total_its; it += S::NG) {
      const int s = it % kStages, d = it % kRing;
      // the TMEM stage's last user has retired (nobody's in the first round, which finds fresh barriers)
      if (!mbar_wait(bar(BAR_MMA_DONE + d), ((it / kRing) & 1) ^ 1u, abort_flag, 0x410 | d)) break;
      if (!mbar_wait(bar(BAR_FULL + s), (it / kStages) & 1, abort_flag, 0x400 | s)) break;
      tc_fence_after();
      const uint8_t* pk = base_ptr + plan.pack + s * kStepPackBytes + np_l * kStepK;
      const uint8_t* sc_tile = base_ptr + plan.scale + s * kStepScaleBytes;
      const uint8_t* zp_tile = base_ptr + plan.zp + s * kStepZpBytes;
      DequantSub<COLWISE, decltype(bsh)::value, decltype(zp)::value != 0, KSUB> sub[KSUB];
#pragma unroll
      for (int u = 0; u < KSUB; ++u) sub[u].load(pk, u, sc_tile, zp_tile, n_l);
#pragma unroll
      for (int u = 0; u < KSUB; ++u) {
        uint32_t out[32];
        sub[u].emit(sc_tile, zp_tile, u, n_l, rot_lo, rot_hi, out);
        tmem_st_32x32b_x32(tmem_row + (uint32_t)(d * kStepCols + u * kDeqCols), out);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar(BAR_STEP_FULL + d));
        mbar_arrive(bar(BAR_PACK_FREE + s));
      }
    }
    });
  }

  if (p.split > 1) {
    // ---- split K: the cluster's CTAs hold one fp32 partial tile each.  Part q owns `slice4` groups of four rows: every
    //      CTA stores the other parts' rows of its partial tile into THEIR shared memory (over the activation
    //      ring, idle once the MMAs of all parts have retired) and then adds up its own rows, in part order, with
    //      all its threads.  Four rows of a column travel as one 16-byte store, laid out [part][row group][column]
    //      so that the lanes of a warp are contiguous on both sides; each part starts with its own rows, so that the parts
    //      of a cluster write to different CTAs at a time; the loops are rolled, because they run a few times per launch from
    //      a cold instruction cache.  Measured on B200 against 4-byte stores from an unrolled loop with a branch per row, us:
    //      M = 16, 4096 x 4096, four parts 8.8 / 7.9; M = 48, 2048 x 1024 6.0 / 4.9; M = 256, 4096 x 4096, four parts 15.7 / 14.9
    //      (16.3 where all parts start with row 0); M = 512, two parts 21.3 / 19.2; M = 300, 8192 x 1024, five parts (and tiles
    //      of one height) 16.9 / 12.8.
    //      With the partial tiles in global memory and one finishing CTA, which read them chunk by
    //      chunk from L2 (one round trip per 32 rows and part), more parts cost more than they gave: K = 4096, N = 1024,
    //      M = 128: four parts through memory 15.4 us, eight 21.7.
    //      A cluster's CTAs are co-resident by construction, so nobody waits for a CTA that is not running.
    asm volatile("griddepcontrol.wait;" ::: "memory");  // all warps store to the output
    __syncwarp();
    cluster_sync_all();  // every part's epilogue warps have seen their accumulator complete
    tc_fence_after();
    const int split = p.split, part = (int)blockIdx.x % split, tile = (int)blockIdx.x / split;
    const Columns col = columns_of<G>(p, tile / p.m_tiles);
    const int n_tile = col.unit, m0 = (tile % p.m_tiles) * p.BM;
    const int rows = min(p.BM, p.M - m0);
    const int slice4 = (p.BM / 4 + split - 1) / split;
    const uint32_t region = base + plan.act;
    if (warp < S::kActProducerWarp) {
      // a warp may read the TMEM lanes of its quarter: the epilogue and dequantizer warps share the columns
      const int n_l = 32 * (warp & 3) + lane;
      const uint32_t lane_base = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16);
      const int inv = slice_inverse(slice4);
      const int chunks = (rows + 15) / 16, first = chunks * part / split;  // BM is a multiple of 16
#pragma unroll 1
      for (int i = warp >> 2; i < chunks; i += S::NG + 1) {
        const int c0 = 16 * (first + i < chunks ? first + i : first + i - chunks);
        uint32_t v[16];
        tmem_ld_32x32b_x16(lane_base + (uint32_t)c0, v);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int r4 = c0 / 4 + g, owner = slice_owner(r4, inv), rg = r4 - owner * slice4;
          st_shared_cluster_v4(map_to_cta(region + (uint32_t)(((part * slice4 + rg) * TILE_N + n_l) * 16), (uint32_t)owner),
                               v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
        }
      }
    }
    cluster_sync_all();
    const int g0 = part * slice4, mine = min(slice4, (rows + 3) / 4 - g0);
    const float4* src = reinterpret_cast<const float4*>(base_ptr + plan.act);
#pragma unroll 1
    for (int idx = threadIdx.x; idx < mine * TILE_N; idx += S::kThreads) {  // whole warps
      const int n = n_tile * TILE_N + (idx % TILE_N);
      float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
      for (int q = 0; q < split; ++q) {
        const float4 f = src[q * slice4 * TILE_N + idx];
        sum.x += f.x;
        sum.y += f.y;
        sum.z += f.z;
        sum.w += f.w;
      }
      // lanes pair up (n even / odd): the even one stores rows 0 and 1 of both columns, the odd one rows 2 and 3
      const int odd = lane & 1;
      const float got0 = __shfl_xor_sync(0xffffffffu, odd ? sum.x : sum.z, 1);
      const float got1 = __shfl_xor_sync(0xffffffffu, odd ? sum.y : sum.w, 1);
      __half2 h0 = odd ? __floats2half2_rn(got0, sum.z) : __floats2half2_rn(sum.x, got0);
      __half2 h1 = odd ? __floats2half2_rn(got1, sum.w) : __floats2half2_rn(sum.y, got1);
      const int m = m0 + 4 * (g0 + idx / TILE_N) + 2 * odd;
      if (n < col.N) {  // N is a multiple of 16: the pair is in or out together
        // the bias is added to the rounded result in fp16, as above
        if (col.bias) {
          const __half2 b = *reinterpret_cast<const __half2*>(col.bias + (n & ~1));
          h0 = __hadd2(h0, b);
          h1 = __hadd2(h1, b);
        }
        __half* dst = col.out + (size_t)m * col.N + (n & ~1);
        if (m < p.M) *reinterpret_cast<__half2*>(dst) = h0;
        if (m + 1 < p.M) *reinterpret_cast<__half2*>(dst + col.N) = h1;
      }
    }
  }

  // ---- teardown ----
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) __nanosleep(50000);  // let copies in flight land
  __syncthreads();
  if (warp == S::kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols)
                 : "memory");
  }
}

#include "blkq4_gemm_tc_pair.cuh"

// ---- host side ---------------------------------------------------------------------------

}  // namespace

namespace {

constexpr int kMaxSplit = 8;  // parts of a tile: the portable cluster size

// Work plan.  The kernel is persistent with one CTA per SM.  A problem with few output tiles
// (prefill of a 4096-wide layer at M = 512: 64 tiles on 148 SMs) leaves SMs idle: cutting every
// tile's K range in `split` work items fills them.  A problem with more tiles than SMs but not a
// whole number of rounds (256 tiles: the second round keeps 108 of 148 SMs busy) is cut in one
// contiguous range of k steps per CTA instead ("balanced", see Params).
struct SplitPlan {
  int split, k_per_item;  // k_per_item steps per part, the last part what is left
  int balanced;
  size_t flags_bytes, total_bytes;  // workspace: [flags, 256-byte aligned][partials]
};

inline int column_tiles(int N) { return (N + TILE_N - 1) / TILE_N; }
inline int column_pairs(int N) { return (column_tiles(N) + 1) / 2; }

SplitPlan plan_split(int M, int n_tiles, int K, size_t ws_bytes_available) {
  const int BM = tile_rows(M, 16);
  const int tiles = ((M + BM - 1) / BM) * n_tiles;
  const int k_steps = (K + step_k(BM) - 1) / step_k(BM);
  const int ws_rows = M >= 256 ? 256 : BM;  // of a partial tile in the workspace: its size is part of the interface
  const int sms = sm_count() > 0 ? sm_count() : 148;
  SplitPlan best{1, k_steps, 0, 0, 0};
  if (tiles > sms) {
    // balanced ranges: every range longer than a tile (a cut tile then has exactly two parts), and only when whole
    // rounds would leave more than a fifth of the SM time idle.  The extra work item and the fp32 exchange cost about
    // 4.5 us, whatever the balance gains.  Measured on B200, whole rounds / balanced, us (K x N):
    //   M = 64, block 128: 8192 x 22528 (176 tiles, 59 % busy) 46.6 / 35.7; 25600 46.7 / 40.4; 28672 (76 %) 47.4 / 44.9;
    //           above the line 32768 (86 %) 50.5 / 52.7; 36864 (97 %) 53.7 / 58.2; 4096 x 22528 24.7 / 20.6; 28672 25.4 / 24.4
    //   M = 128: 8192 x 22528 56.2 / 48.3; 28672 60.5 / 58.9; 32768 65.9 / 66.3
    //   M = 16, block 32: 8192 x 22528 44.4 / 31.5; 28672 44.8 / 38.5; 30720 (81 %, not taken) 45.1 / 40.7
    // With few steps a tile the line comes too late: K = 2048, M = 64, N = 28672 14.7 / 15.8; M = 128, 4096 x 28672 31.3 / 32.4.
    const int rounds = (tiles + sms - 1) / sms;
    const long long total_steps = (long long)tiles * k_steps;
    static const bool off = getenv("BLKQ4_TC_NO_BALANCE") != nullptr;
    if (!off && total_steps < (1ll << 30) / sms && total_steps / sms >= k_steps + 2 * min_part(step_k(BM)) &&
        (double)tiles < 0.80 * rounds * sms) {
      const size_t flags = ((size_t)sms * sizeof(unsigned) + 255) & ~(size_t)255;
      const size_t total = flags + (size_t)sms * ws_rows * TILE_N * sizeof(float);
      if (total <= ws_bytes_available) best = SplitPlan{1, k_steps, 1, flags, total};
    }
    return best;
  }
  // Split only when every work item still gets an SM of its own (one round).  The parts exchange their partial tiles
  // through distributed shared memory, so they may be uneven and as many (of at least 512 k) as there are SMs for.
  // The workspace is the caller's opt-in (a split changes the order of the fp32 sums) and is not touched.  Its size is
  // part of the interface - which calls split, and which the static-scratch entry refuses - and stays what it was
  // when the parts met there: the fp32 partial tiles of an even two- or four-way split, or one page of flags where K
  // does not divide evenly.  A smaller one gets the split it would hold.  Up to 16 rows no opt-in is asked for:
  // those calls never needed one.
  auto even_split = [&](size_t avail, size_t* bytes) {
    int split = 1;
    *bytes = 0;
    for (int parts = 2; parts <= 4; parts *= 2) {
      const size_t flags = ((size_t)tiles * sizeof(unsigned) + 255) & ~(size_t)255;
      const size_t total = flags + (size_t)tiles * (parts - 1) * ws_rows * TILE_N * sizeof(float);
      if (k_steps % parts != 0 || (k_steps / parts) * step_k(BM) < 512 || tiles * parts > sms || total > avail) continue;
      split = parts;
      *bytes = total;
    }
    return split;
  };
  size_t bytes = 0, all_bytes = 0;
  const int fits = even_split(ws_bytes_available, &bytes), wanted = even_split(~(size_t)0, &all_bytes);
  const bool free_split = M <= 16;
  if (!free_split && fits < wanted) return SplitPlan{fits, k_steps / fits, 0, 0, bytes};
  if (!free_split && ws_bytes_available < 256) return best;
  for (int parts = 2; parts <= kMaxSplit; ++parts) {
    const int per = (k_steps + parts - 1) / parts;
    const int split = (k_steps + per - 1) / per;  // no empty part
    if (split == 1 || per * step_k(BM) < 512 || tiles * split > sms) continue;
    best = SplitPlan{split, per, 0, 0, free_split ? 0 : bytes ? bytes : 256};
  }
  return best;
}

// The one-CTA kernel for tiles of BM rows and `steps` pipeline steps a CTA.
template <int G>
using Kern = void (*)(CUtensorMap, WeightMaps<G>, Params);
template <int G>
struct KernelChoice {
  Kern<G> kern;
  int threads, which;  // which: index of the per-device caches
  size_t smem;
  int deq_cols;        // tensor memory of the dequantized stages
};
std::atomic<int> g_granted_smem[16][64];

template <int G>
KernelChoice<G> choose_kernel(bool colwise, int BM, int steps = 0) {
  KernelChoice<G> c;
  auto pick = [&](auto shape, int idx) {
    using S = decltype(shape);
    c.kern = colwise ? (Kern<G>)gemm_tc_kernel<true, S, G> : (Kern<G>)gemm_tc_kernel<false, S, G>;
    c.threads = S::kThreads;
    c.which = 4 * idx + (G > 1 ? 2 : 0) + (colwise ? 1 : 0);
    c.smem = make_plan(S::MAXM, S::WS, S::RING, S::KSUB).total;
    c.deq_cols = S::kDeqTmemCols;
  };
  if (BM <= ShapeSmall::MAXM && steps >= kLongSteps) pick(ShapeSmallLong{}, 3);
  else if (BM <= ShapeSmall::MAXM) pick(ShapeSmall{}, 0);
  else if (BM <= ShapeMid::MAXM) pick(ShapeMid{}, 1);
  else pick(ShapeLarge{}, 2);
  return c;
}

// Clusters of `split` CTAs of the kernel that are resident at once on the current device, 0 when it cannot say.
template <int G>
int resident_clusters(const KernelChoice<G>& kc, int split) {
  static std::atomic<int> cache[16][kMaxSplit + 1][64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const bool cached = dev >= 0 && dev < 64;
  int n = cached ? cache[kc.which][split][dev].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sm_count() / split * split);
  cfg.blockDim = dim3(kc.threads);
  cfg.dynamicSmemBytes = kc.smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (ensure_dynamic_smem(kc.kern, kc.smem, g_granted_smem[kc.which]) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kc.kern, &cfg) != cudaSuccess || n < 0) {
    cudaGetLastError();
    return 0;
  }
  if (cached && n > 0) cache[kc.which][split][dev].store(n, std::memory_order_relaxed);
  return n;
}

// A group of SMs holds whole clusters only, so fewer than SMs / split may fit: cut in fewer parts until all
// clusters of the problem run in one round.
template <int G>
void fit_split(const KernelChoice<G>& kc, int tiles, int k_steps, SplitPlan& sp) {
  while (sp.split > 1 && resident_clusters(kc, sp.split) < tiles) {
    sp.k_per_item = (k_steps + sp.split - 2) / (sp.split - 1);
    sp.split = (k_steps + sp.k_per_item - 1) / sp.k_per_item;
  }
}

// Whether there is a device to ask for its clusters.
bool have_device() {
  int devices = 0;
  if (cudaGetDeviceCount(&devices) != cudaSuccess) cudaGetLastError();
  return devices > 0;
}

// The kernel of a planned launch; the plan's split as this device can run it.
template <int G>
KernelChoice<G> fit_plan(bool colwise, int BM, int tiles, int k_steps, int sms, SplitPlan& sp) {
  const int cta_steps = sp.split > 1 ? sp.k_per_item : (int)((long long)tiles * k_steps / (tiles < sms ? tiles : sms));
  const KernelChoice<G> kc = choose_kernel<G>(colwise, BM, cta_steps);
  fit_split(kc, tiles, k_steps, sp);
  return kc;
}

}  // namespace

namespace {

// Plan of the CTA-pair kernel (blkq4_gemm_tc_pair.cuh): two CTAs per 256 (weight columns) x BM tile, each
// staging half of the activation rows; the pair's UMMA N = BM must be a multiple of 32.  Used for
// M >= 256 when the pair tiles fill at least one round of the device's pairs (the pair kernel has no
// split-K: M = 512 on a 4096-wide layer, 32 pair tiles, runs faster split over single CTAs).  With a
// workspace, and when whole rounds would idle more than a fifth of the pairs' time, the work is cut in
// balanced ranges.  Measured on B200, whole rounds / balanced: 86 pair tiles on 74 pairs (M = 512, 4096 -> 11008)
// 45.3 / 42.5 us; 156 tiles (M = 512, N = 19968) 78 / 70; 100 tiles (N = 12800) 46.5 / 47.8; 112 tiles (M = 256,
// K = 8192, N = 28672) 96.2 / 96.7; above the line 128 tiles (M = 2048, N = K = 4096, 86 % busy in whole rounds)
// 51.8 / 60.4 and 448 tiles (M = 1024, K = 8192, N = 28672) 332 / 338: one more accumulator hand-over per pair and the
// fp32 exchange of a 128 KB partial tile per CTA cost what the balance gains there.
struct PairPlan {
  bool use;
  int BM, m_tiles, items, balanced;
  size_t flags_bytes, total_bytes;
};

PairPlan plan_pair(int M, int n_pairs, int K, size_t ws_bytes_available) {
  static const bool pair_off = getenv("BLKQ4_TC_NO_PAIR") != nullptr;
  static const int pair_min_m = getenv("BLKQ4_TC_PAIR_MIN_M") ? atoi(getenv("BLKQ4_TC_PAIR_MIN_M")) : 256;
  static const double balance_below =
      getenv("BLKQ4_TC_PAIR_BALANCE_BELOW") ? atof(getenv("BLKQ4_TC_PAIR_BALANCE_BELOW")) : 0.80;
  PairPlan pl{false, 0, 0, 0, 0, 0, 0};
  if (M < pair_min_m || pair_off) return pl;
  const int sms = sm_count() > 0 ? sm_count() : 148;
  const int pairs = sms / 2;
  pl.BM = tile_rows(M, 32);
  pl.m_tiles = (M + pl.BM - 1) / pl.BM;
  pl.items = pl.m_tiles * n_pairs;
  const int k_steps = K / BLOCK_K;
  const long long total_steps = (long long)pl.items * k_steps;
  const int rounds = (pl.items + pairs - 1) / pairs;
  static const bool balance_off = getenv("BLKQ4_TC_NO_BALANCE") != nullptr;
  // Fewer tiles than pairs: the one-CTA kernel splits K.  (The pair kernel can do it too - ranges shorter
  // than a tile, a tile finished from several partial tiles - but measured slower: M = 512, K = N = 4096
  // 34.5 vs 20.9 us, K = 11008 50.9 vs 40.1 us; a 128 KB fp32 partial tile per CTA is a dear exchange.)
  if (pl.items < pairs) return pl;
  // Balanced ranges need a workspace (one flag word and one fp32 partial tile per CTA), ranges of at least
  // eight steps, and pay when whole rounds would idle more than a fifth of the pairs' time.
  const size_t flags = ((size_t)sms * sizeof(unsigned) + 255) & ~(size_t)255;
  const size_t total = flags + (size_t)sms * (M >= 256 ? 256 : pl.BM) * TILE_N * sizeof(float);  // part of the interface
  const bool can_balance = !balance_off && total_steps < (1ll << 30) / pairs && total_steps / pairs >= 8 &&
                           (double)pl.items < balance_below * rounds * pairs && total <= ws_bytes_available;
  pl.use = true;
  if (can_balance) {
    pl.balanced = 1;
    pl.flags_bytes = flags;
    pl.total_bytes = total;
  }
  return pl;
}

// What a problem is launched as.
//
// plan_pair and plan_split make tiles as high as they can be (each weight is dequantized once per 256 rows) and then cut K
// until the SMs are busy.  That is right for long K.  With fewer than 48 steps a tile is short, and what it costs besides
// its steps - filling the pipeline, draining the accumulator by four warps, above all a cluster's or two ranges' exchange of fp32
// partial tiles - outweighs the second conversion of the weights: more and lower tiles, each with all or more of K, are faster.
// Below kCostK the parts of K follow short_k_parts and the height of the tiles is the one that promises the largest gain, where
// both column-wise and row-wise blocks gain (the conversion of row-wise ones takes longer, and a plan serves all blockings).
// Measured on B200 (block 64, zero points), tiles as high and parts as many as possible / as planned here, us (M, K x N): 256,
// 512 x 512 6.4 / 3.5 (64 rows); 256, 1024 x 1024 9.6 / 4.4 (64); 512, 1024 x 4096 11.2 / 7.4 (128); 23, 1024 x 7328 0.71 of the
// time in one part instead of two; 128, 1024 x 28672 14.9 / 10.6; 469, 960 x 576 9.3 / 6.1; 320, 512 x 22528 18.2 / 12.8 (tiles
// of the one-CTA kernel instead of balanced ranges of pairs); 512, 2048 x 2048 11.9 / 8.8.  Over 394 random problems of 17 to 1100
// rows and 512 to 3008 k the planned launch takes 0.90 of the time, 0.93 with row-wise blocks of 32 (the best candidate of each 0.85
// and 0.90); two and five of them are slower by more than 3 %.  From 3072 to 4095 k the gain was 2.6 %, above 2 %, within
// the prediction's error: plans stay as they are there.  Pair tiles in whole rounds are not questioned: one-CTA tiles took
// 0.82 to 1.13 of their time.
constexpr int kCostK = 3072, kMinPlannedRows = 48;

// Parts of K of a problem that plan_split would cut in `parts`.  Up to 64 rows, where lower tiles do not help, a split in two
// costs more than it gains below 2048 k (whole / in two: K = 832 to 1088 0.68 to 0.90, 1856 0.83, 2048 0.92, 2496 1.00), one in
// four does not (1.0 to 1.4); above, only five or more parts say that the SMs would stay idle with low tiles too.  Fewer than eight
// column tiles leave them idle in any case: those keep their parts.
// The columns count through `parts`, which is what fills the SMs with high tiles, and through that limit: layers of one K can be cut
// otherwise than a group of them, and gemm_tc_group_keeps_bits says which may share a launch.
inline int short_k_parts(int M, int n_tiles, int K, int parts) {
  if (n_tiles < 8) return parts;
  if (M <= 64) return parts >= 3 || K >= 2048 ? parts : 1;
  return parts >= 5 ? 4 : 1;
}

// Predicted time in us, by least squares over the candidates of the problems above (rms error 10 %): start-up, then per round of
// tiles the 64-k steps of one and its end, then the exchange between the parts of a cluster or of balanced ranges.
// The constants are the kernels': after a change of their steps or ends they are fitted again, by timing every height of compute_plan's
// loop, and plan_high_tiles, on random problems in its range (graphs of launches with the early weight fetch; blocks of 64 with zero
// points column-wise, of 32 row-wise) and least squares of the relative error over the terms of one_cta and balanced_pairs.
struct TileCost {
  double start, step, step_row, end, end_row;
};
struct CostModel {
  TileCost small, mid, large, pair;
  double split, split_row, split_part, balanced;
  double us(const TileCost& c, int BM, double rounds, int steps64) const {
    return c.start + rounds * (steps64 * (c.step + c.step_row * BM) + c.end + c.end_row * BM);
  }
  double one_cta(int BM, int tiles, const SplitPlan& sp, int sms) const {
    const TileCost& c = BM <= ShapeSmall::MAXM ? small : BM <= ShapeMid::MAXM ? mid : large;
    const double rounds = sp.balanced ? (double)tiles / sms : (double)((tiles * sp.split + sms - 1) / sms);
    return us(c, BM, rounds, sp.k_per_item * (step_k(BM) / BLOCK_K)) +
           (sp.balanced ? balanced : sp.split > 1 ? split + split_row * BM + split_part * sp.split : 0.0);
  }
  double balanced_pairs(int BM, int items, int pairs, int steps64) const {
    return us(pair, BM, items / (double)pairs, steps64) + balanced;
  }
};
constexpr CostModel kColumnWise{{1.5869, 0.165, 0, 0.6429, 0},
                               {2.272, 0.1311, 0.0004, 0, 0.0083},
                               {1.4118, 0.1161, 0.0009, 0, 0.0098},
                               {5.4188, 0.1224, 0.0009, 0, 0.003},
                               1.13, 0.0071, 0.21, 6.6},
    kRowWise{{0.8339, 0.2595, 0, 0.5351, 0},
             {1.6446, 0.219, 0.0004, 0, 0.0074},
             {1.2523, 0.2433, 0.0005, 0, 0.0096},
             {5.7228, 0.2428, 0.0007, 0, 0.0019},
             1.42, 0.0048, 0.29, 6.3};

struct TcPlan {
  bool pair;
  PairPlan pp;   // pair
  int BM;        // rows of a tile, either kernel
  int m_tiles;
  SplitPlan sp;  // !pair
};

// plan_pair and plan_split as they are.
TcPlan plan_high_tiles(int M, int n_tiles, int n_pairs, int K, size_t ws_bytes_available) {
  TcPlan pl{};
  pl.pp = plan_pair(M, n_pairs, K, ws_bytes_available);
  pl.pair = pl.pp.use;
  pl.BM = pl.pair ? pl.pp.BM : tile_rows(M, 16);
  pl.m_tiles = (M + pl.BM - 1) / pl.BM;
  if (!pl.pair) pl.sp = plan_split(M, n_tiles, K, ws_bytes_available);
  return pl;
}

TcPlan compute_plan(int M, int n_tiles, int n_pairs, int K, size_t ws_bytes_available, bool gather) {
  TcPlan pl = plan_high_tiles(M, n_tiles, n_pairs, K, gather ? 0 : ws_bytes_available);
  if (gather || M <= 16 || K >= kCostK || (pl.pair && !pl.pp.balanced)) return pl;
  const int sms = sm_count() > 0 ? sm_count() : 148;
  const int parts = pl.pair ? 1 : short_k_parts(M, n_tiles, K, pl.sp.split);
  auto high_us = [&](const CostModel& c) {
    return pl.pair ? c.balanced_pairs(pl.BM, pl.pp.items, sms / 2, K / BLOCK_K) : c.one_cta(pl.BM, pl.m_tiles * n_tiles, pl.sp, sms);
  };
  const double high_col = high_us(kColumnWise), high_row = high_us(kRowWise);
  // the gain has to exceed the prediction's error: against the same kernel, and against the other one
  double best = pl.pair ? 0.88 : 0.96;
  int last_rows = 0;
  for (int m_tiles = (M + 255) / 256;; ++m_tiles) {
    const int BM = ((M + m_tiles - 1) / m_tiles + 15) / 16 * 16;
    if (BM < kMinPlannedRows && last_rows > 0) break;
    if (BM == last_rows) {
      if (BM <= kMinPlannedRows) break;
      continue;
    }
    last_rows = BM;
    const int tiles = (M + BM - 1) / BM * n_tiles, k_steps = (K + step_k(BM) - 1) / step_k(BM);
    const int per = (k_steps + parts - 1) / parts;
    if ((k_steps + per - 1) / per != parts || (parts > 1 && tiles * parts > sms)) continue;
    const SplitPlan sp{parts, per, 0, 0, 0};
    const double col = kColumnWise.one_cta(BM, tiles, sp, sms) / high_col, row = kRowWise.one_cta(BM, tiles, sp, sms) / high_row;
    const double ratio = col > row ? col : row;
    if (ratio >= best) continue;
    best = ratio;
    pl.pair = false;
    pl.BM = BM;
    pl.m_tiles = (M + BM - 1) / BM;
    pl.sp = sp;
  }
  return pl;
}

// gather: the fused exchange, which lives in the pair kernel's epilogue and runs in whole rounds.
// A plan is a function of the arguments and the number of SMs; a model asks for the same few again and again, and a search takes up to
// half a microsecond of the launch: the latest ones are kept, per thread and direct-mapped, as the tensor maps are.
TcPlan plan_tc(int M, int n_tiles, int n_pairs, int K, size_t ws_bytes_available, bool gather = false) {
  struct Entry {
    int M, n_tiles, n_pairs, K, sms;
    size_t ws;
    bool gather;
    TcPlan plan;
  };
  constexpr int kEntries = 64;
  thread_local Entry cache[kEntries];  // M == 0: empty
  const int sms = sm_count();
  Entry& e = cache[((uint32_t)M * 31u + (uint32_t)n_tiles * 7u + (uint32_t)K / 64u) % kEntries];
  if (M <= 0 || e.M != M || e.n_tiles != n_tiles || e.n_pairs != n_pairs || e.K != K || e.sms != sms || e.ws != ws_bytes_available ||
      e.gather != gather)
    e = Entry{M, n_tiles, n_pairs, K, sms, ws_bytes_available, gather, compute_plan(M, n_tiles, n_pairs, K, ws_bytes_available, gather)};
  return e.plan;
}

}  // namespace

size_t gemm_tc_workspace_bytes(int M, int N, int K) {
  if (M <= 16) return 0;
  const PairPlan pp = plan_pair(M, column_pairs(N), K, ~(size_t)0);
  if (pp.use) return pp.total_bytes;
  return plan_split(M, column_tiles(N), K, ~(size_t)0).total_bytes;
}

// Which problems of up to 16 rows run here rather than on the generic skinny kernel (blkq4_gemv.cu): both convert
// the weights to fp16 by the same formula and sum in fp32.  Only those whose blocking no other skinny kernel takes
// (row-wise, or blocks of 16 and 32): the others scale fp32 sums instead, which is more accurate.  (Of the problems that stay
// there, the decode kernel has since taken the column-wise ones of a few rows: small_blocks_are_faster of blkq4_gemv_stream.cu.)
// Measured on B200 (graphs of launches over 512 MB of weights), generic against this one, us, K x N, block 32 column-wise
// with zero points (row-wise).  Blocks of 16, and row-wise blocks of 128, lie within 5 % of these.
//   M = 1:  4096 x 8192 13.4 / 10.9 (15.3 / 13.7);  8192 x 512 10.0 / 6.1 (13.1 / 7.0);  8192 x 4096 12.2 / 11.3 (14.8 / 14.1);
//           2048 x 16384 13.7 / 8.8 (16.2 / 11.5);  4096 x 11008 16.9 / 13.5 (20.7 / 18.5);  8192 x 28672 66.6 / 39.7
//           (80.0 / 55.4);  not taken: 2048 x 4096 5.0 / 6.6 (5.5 / 7.3);  4096 x 4096 7.5 / 8.1 (8.7 / 9.6)
//           M = 2, 4 and 8: within 8 % of M = 1 on either side, the generic kernel slower with M (8192 x 28672: 77.4 / 40.1)
//   M = 16: 512 x 2048 5.7 / 3.3 (5.7 / 3.3);  1536 x 4096 8.0 / 6.5 (8.7 / 7.0);  2048 x 2048 6.3 / 5.3 (7.0 / 5.6);
//           4096 x 4096 10.9 / 8.5 (11.7 / 10.0);  2048 x 11008 12.7 / 8.1 (13.8 / 10.3, not taken);
//           4096 x 11008 22.2 / 13.6 (25.3 / 18.6);  8192 x 28672 81.1 / 40.3 (88.2 / 55.8);  M = 9, 12: within 3 % of M = 16
// The generic kernel is at its best at K = 1024 and 2048, where each of its warps has its minimum of four 64-k steps and no
// more, and where N just fills its rounds of 32 columns per SM; there the cluster exchange here costs more than it
// gains.  M = 16:
//   2048 x 4096 6.6 / 7.0 (7.4 / 7.8);  4608 6.7 / 7.4 (7.5 / 8.4);  5120 8.1 / 7.5 (8.4 / 8.7);  7168 8.2 / 8.0 (8.6 / 9.3)
//   1024 x 512 5.0 / 5.2 (5.0 / 5.2);  1024 5.2 / 5.2 (5.1 / 5.3);  8192 6.6 / 6.8 (7.3 / 7.4);  9216 6.7 / 7.1 (7.3 / 7.8);
//   11008 7.3 / 5.2 (7.9 / 6.0)
// Elsewhere the slower side is taken by 7 % at most (row-wise 2560 x 7168 10.0 / 10.5, with blocks of 128 9.7 / 10.4).
bool gemm_tc_takes_skinny(int block, bool colwise, int M, int N, int K, const void* scales, const void* zp) {
  if (M > 16 || (colwise && block >= 64)) return false;
  if (reinterpret_cast<uintptr_t>(scales) % 16 != 0 || reinterpret_cast<uintptr_t>(zp) % 16 != 0) return false;
  const long long kn = (long long)K * N;
  if (M <= 8) return K >= 8192 || kn >= (1ll << 25);
  const int round = 32 * (sm_count() > 0 ? sm_count() : 148);  // columns per round of the generic kernel
  if (K == 2048 && N > round * 4 / 5 && (N <= round || !colwise)) return false;
  if (K == 1024 && ((N > round * 17 / 10 && N <= 2 * round) || (N <= 1024 && !colwise))) return false;
  return !(N >= 8192 && K >= 2048 && kn <= (colwise ? 1ll << 24 : 1ll << 25));
}

size_t gemm_tc_workspace_bytes_any(int block, bool colwise, int M, int N, int K) {
  if (M > 16) return gemm_tc_workspace_bytes(M, N, K);
  return gemm_tc_takes_skinny(block, colwise, M, N, K, nullptr, nullptr) ? plan_split(M, column_tiles(N), K, ~(size_t)0).total_bytes : 0;
}

bool gemm_tc_split_plan_refusable(int M, int N, int K, size_t capacity) {
  if (M <= 16) return false;
  const SplitPlan sp = plan_split(M, column_tiles(N), K, ~(size_t)0);
  return sp.total_bytes > capacity && sp.balanced == 0;
}

bool gemm_tc_gather_supported(int M, int N, int K) {
  return M > 16 && plan_pair(M, column_pairs(N), K, 0).use;
}

bool gemm_tc_plan_balanced(int M, int N, int K) {
  if (M <= 16) return false;
  const PairPlan pp = plan_pair(M, column_pairs(N), K, ~(size_t)0);
  if (pp.use) return pp.balanced != 0;
  return plan_split(M, column_tiles(N), K, ~(size_t)0).balanced != 0;
}

namespace {

// G == 1: one weight matrix.  G > 1: the `grp` of them, whose tiles the plans see as those of one wide matrix.
template <int G>
std::string launch_weights(int block, bool colwise, int M, int K, cudaStream_t stream, const __half* a, const GemmGroup& grp,
                           void* workspace, size_t workspace_bytes, unsigned flags, const GatherTable* gt) {
  Params p{};
  if (gt) p.gt = *gt;
  const int N = grp.n[0];
  const uint8_t* zp = grp.zp[0];
  int n_tiles = 0, n_pairs = 0;
  for (int i = 0; i < grp.count; ++i) {
    n_tiles += column_tiles(grp.n[i]);
    n_pairs += column_pairs(grp.n[i]);
  }
  p.M = M; p.N = N; p.K = K; p.block = block;
  p.block_shift = block == 16 ? 4 : block == 32 ? 5 : block == 64 ? 6 : 7;
  const bool ws_ok = workspace && reinterpret_cast<uintptr_t>(workspace) % 256 == 0;
  // the fused exchange lives in the pair kernel's epilogue and runs in whole rounds
  const TcPlan plan = plan_tc(M, n_tiles, n_pairs, K, ws_ok ? workspace_bytes : 0, gt != nullptr);
  const bool pair = plan.pair;
  if (gt && !pair) return "unsupported shape for the fused all-gather";
  p.BM = plan.BM;
  p.m_tiles = plan.m_tiles;
  p.n_tiles = n_tiles;
  p.has_zp = zp != nullptr;
  p.out = grp.out[0];
  p.bias = grp.bias[0];
  // tensor memory of the one-CTA kernel: accumulators first, then the dequantized stages
  const int deq_cols = choose_kernel<G>(colwise, p.BM).deq_cols;
  p.acc_bufs = (2 * p.BM + deq_cols <= 512) ? 2 : 1;
  p.a_col0 = p.acc_bufs * p.BM;
  {
    const uint32_t need = (uint32_t)(p.a_col0 + deq_cols);
    p.tmem_cols = 32;
    while (p.tmem_cols < need) p.tmem_cols <<= 1;
  }

  if constexpr (G > 1) {
    p.grp = grp;
    int end = 0;
    for (int i = 0; i < grp.count; ++i) {
      end += pair ? column_pairs(grp.n[i]) : column_tiles(grp.n[i]);
      p.grp.tile_end[i] = end;
    }
  }

  // k per pipeline step: the box of the weights and of the meta spans it, the activations come in 64-k tiles
  const int sk = pair ? BLOCK_K : step_k(p.BM);
  CUtensorMap tm_act;
  WeightMaps<G> wm;
  bool ok = encode_tensor_map_2d(&tm_act, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a, (uint64_t)K, (uint64_t)M, BLOCK_K,
                      pair ? (uint32_t)(p.BM / 2) : (uint32_t)p.BM, CU_TENSOR_MAP_SWIZZLE_128B);
  if (colwise) {
    p.meta_rows = block >= sk ? 1 : sk / block;
    p.meta_row_bytes_s = TILE_N * 2;
    p.meta_row_bytes_z = TILE_N;
  } else {
    p.meta_rows = block >= TILE_N ? 1 : TILE_N / block;
    p.meta_row_bytes_s = (uint32_t)sk * 2;
    p.meta_row_bytes_z = (uint32_t)sk;
  }
  for (int i = 0; i < grp.count; ++i) {
    const int Ni = grp.n[i];
    // Packed tiles of 128-byte rows carry the 128-byte swizzle: the dequantizers' 16-byte loads of eight
    // neighbouring packed columns would otherwise all fall on the same banks.
    // No swizzle on 64-byte rows: the dequantizers' 16-byte loads of eight neighbouring packed
    // columns (64 bytes apart) do conflict four ways, but a 64-byte TMA swizzle that removes the
    // conflicts measured 1-2 % SLOWER on the same GPU (M = 2048, 4096 x 4096: 59.2 vs 58.2 us): those loads are not on
    // the critical path, the extra XOR per load is.
    ok = ok && encode_tensor_map_2d(&wm.pack[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, grp.packed[i], (uint64_t)K, (uint64_t)(Ni / 2),
                         (uint32_t)sk, TILE_N / 2, sk == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE);
    const uint64_t cols = colwise ? (uint64_t)Ni : (uint64_t)K, rows = (uint64_t)((colwise ? K : Ni) / block);
    const uint32_t box = colwise ? (uint32_t)TILE_N : (uint32_t)sk;
    ok = ok && encode_tensor_map_2d(&wm.scale[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, grp.scales[i], cols, rows, box,
                                    (uint32_t)p.meta_rows, CU_TENSOR_MAP_SWIZZLE_NONE);
    ok = ok && encode_tensor_map_2d(&wm.zp[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, zp ? grp.zp[i] : grp.packed[i], cols, rows, box,
                                    (uint32_t)p.meta_rows, CU_TENSOR_MAP_SWIZZLE_NONE);
  }
  if (!ok) return "cuTensorMapEncodeTiled failed";

  const int sms = sm_count();
  if (pair) {
    p.k_steps = K / BLOCK_K;
    const PairPlan& pp = plan.pp;
    p.num_items = pp.items;
    p.n_pairs = n_pairs;
    // fused all-gather: walk the column pairs of one m tile together, so that at any moment the stores of all
    // ranks fall into a few hundred rows of every destination
    static const bool nf_off = getenv("BLKQ4_TC_GATHER_M_FASTEST") != nullptr;
    p.n_fastest = (gt && !nf_off) ? 1 : 0;
    static const bool bulk_off = getenv("BLKQ4_TC_GATHER_NO_BULK") != nullptr;
    p.gather_bulk = (gt && !bulk_off) ? 1 : 0;
    p.balanced = pp.balanced;
    p.total_steps = pp.balanced ? pp.items * p.k_steps : 0;
    p.ws_flags = reinterpret_cast<unsigned*>(workspace);
    p.ws_partials = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(workspace) + pp.flags_bytes);
    auto kern = colwise ? gemm_tc_pair_kernel<true, kPairWeightStages, G> : gemm_tc_pair_kernel<false, kPairWeightStages, G>;
    const SmemPlan smem = make_plan(kPairRows, kPairWeightStages, kPairActStages, 1, kPairOutBytes);
    static std::atomic<int> granted[2][64];
    cudaError_t e = ensure_dynamic_smem(kern, smem.total, granted[colwise ? 1 : 0]);
    if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = smem.total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    // pairs that can be resident at once (the cluster size is part of the kernel): one per two SMs at best
    static std::atomic<int> max_pairs[2][64];
    int dev = 0;
    cudaGetDevice(&dev);
    int pairs = (dev >= 0 && dev < 64) ? max_pairs[colwise ? 1 : 0][dev].load(std::memory_order_relaxed) : 0;
    if (pairs <= 0) {
      cfg.gridDim = dim3(sms & ~1);
      cfg.numAttrs = 0;
      int n = 0;
      e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
      if (e != cudaSuccess || n <= 0) { cudaGetLastError(); n = sms / 2; }
      pairs = n < sms / 2 ? n : sms / 2;
      if (dev >= 0 && dev < 64) max_pairs[colwise ? 1 : 0][dev].store(pairs, std::memory_order_relaxed);
    }
    cfg.numAttrs = (flags & BLKQ4_GEMM_EARLY_WEIGHT_FETCH) ? 1 : 0;
    // balanced ranges use every resident pair, whole rounds at most one pair per tile
    cfg.gridDim = dim3(2 * ((p.balanced || p.num_items >= pairs) ? pairs : p.num_items));
    e = cudaLaunchKernelEx(&cfg, kern, tm_act, wm, p);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
    return std::string();
  }
  const int num_tiles = p.m_tiles * p.n_tiles;
  p.k_steps = (K + sk - 1) / sk;
  SplitPlan sp = plan.sp;
  const KernelChoice<G> kc = fit_plan<G>(colwise, p.BM, num_tiles, p.k_steps, sms, sp);
  p.split = sp.split;  // split > 1: at most one item per SM
  p.k_per_item = sp.k_per_item;
  p.min_part = min_part(sk);
  p.balanced = sp.balanced;
  p.total_steps = sp.balanced ? num_tiles * p.k_steps : 0;
  p.ws_flags = reinterpret_cast<unsigned*>(workspace);
  p.ws_partials = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(workspace) + sp.flags_bytes);
  cudaError_t e = ensure_dynamic_smem(kc.kern, kc.smem, g_granted_smem[kc.which]);
  if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kc.threads);
  cfg.dynamicSmemBytes = kc.smem;
  cfg.stream = stream;
  // BLKQ4_GEMM_EARLY_WEIGHT_FETCH: programmatic stream serialization, see the kernel's entry
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  p.num_items = num_tiles * p.split;
  cfg.gridDim = dim3(p.num_items < sms ? p.num_items : sms);
  cfg.attrs = p.split > 1 ? attr : attr + 1;
  cfg.numAttrs = (p.split > 1 ? 1 : 0) + ((flags & BLKQ4_GEMM_EARLY_WEIGHT_FETCH) ? 1 : 0);
  e = cudaLaunchKernelEx(&cfg, kc.kern, tm_act, wm, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
  return std::string();
}

}  // namespace

std::string launch_gemm_tc(int block, bool colwise, int M, int N, int K, cudaStream_t stream,
                           const __half* a, const uint8_t* packed, const __half* scales,
                           const uint8_t* zp, __half* out, const __half* bias, void* workspace,
                           size_t workspace_bytes, unsigned flags, const GatherTable* gt) {
  GemmGroup one{};
  one.count = 1;
  one.n[0] = N;
  one.packed[0] = packed;
  one.scales[0] = scales;
  one.zp[0] = zp;
  one.out[0] = out;
  one.bias[0] = bias;
  return launch_weights<1>(block, colwise, M, K, stream, a, one, workspace, workspace_bytes, flags, gt);
}

std::string launch_gemm_tc_group(int block, bool colwise, int M, int K, cudaStream_t stream, const __half* a,
                                 const GemmGroup& grp, void* workspace, size_t workspace_bytes, unsigned flags) {
  return launch_weights<kMaxGroup>(block, colwise, M, K, stream, a, grp, workspace, workspace_bytes, flags, nullptr);
}

size_t gemm_tc_group_workspace_bytes(int M, int K, int count, const int* n) {
  int n_tiles = 0, n_pairs = 0;
  for (int i = 0; i < count; ++i) {
    n_tiles += column_tiles(n[i]);
    n_pairs += column_pairs(n[i]);
  }
  const PairPlan pp = plan_pair(M, n_pairs, K, ~(size_t)0);
  return pp.use ? pp.total_bytes : plan_split(M, n_tiles, K, ~(size_t)0).total_bytes;
}

namespace {

// K split of a plan as the device runs it, k_per_item in k; 0 where balanced ranges would cut its tiles.
template <int G>
SplitPlan launched_split(bool colwise, int K, int n_tiles, const TcPlan& pl) {
  if (pl.pair) return SplitPlan{1, pl.pp.balanced ? 0 : K, 0, 0, 0};
  SplitPlan sp = pl.sp;
  if (sp.balanced) return SplitPlan{1, 0, 0, 0, 0};
  const int k_steps = (K + step_k(pl.BM) - 1) / step_k(pl.BM);
  if (have_device()) fit_plan<G>(colwise, pl.BM, pl.m_tiles * n_tiles, k_steps, sm_count() > 0 ? sm_count() : 148, sp);
  return SplitPlan{sp.split, sp.split > 1 ? sp.k_per_item * step_k(pl.BM) : K, 0, 0, 0};
}

}  // namespace

// With all the workspace that is asked for.  Layers that high tiles would cut in balanced ranges, or in other parts than their
// group, stay apart although lower tiles may cut all of them alike: which layers share a launch is part of the interface.
bool gemm_tc_group_keeps_bits(bool colwise, int M, int K, int count, const int* n) {
  int n_tiles = 0, n_pairs = 0;
  for (int i = 0; i < count; ++i) {
    n_tiles += column_tiles(n[i]);
    n_pairs += column_pairs(n[i]);
  }
  auto split_of = [&](auto g, int tiles, int pairs, bool high) {
    const TcPlan pl = high ? plan_high_tiles(M, tiles, pairs, K, ~(size_t)0) : plan_tc(M, tiles, pairs, K, ~(size_t)0);
    return launched_split<decltype(g)::value>(colwise, K, tiles, pl);
  };
  const std::integral_constant<int, kMaxGroup> group{};
  const std::integral_constant<int, 1> alone{};
  const SplitPlan all = split_of(group, n_tiles, n_pairs, false), all_high = split_of(group, n_tiles, n_pairs, true);
  if (all.k_per_item == 0) return false;
  for (int i = 0; i < count; ++i) {
    const int tiles = column_tiles(n[i]), pairs = column_pairs(n[i]);
    const SplitPlan one = split_of(alone, tiles, pairs, false), one_high = split_of(alone, tiles, pairs, true);
    if (one.split != all.split || one.k_per_item != all.k_per_item) return false;
    if (one_high.split != all_high.split || one_high.k_per_item == 0) return false;
  }
  return true;
}

int clear_gemm_tc_error(cudaStream_t stream) {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_gemm_tc_error) != cudaSuccess) return -1;
  return cudaMemsetAsync(p, 0, sizeof(int), stream) == cudaSuccess ? 0 : -1;
}

int read_gemm_tc_error(cudaStream_t stream) {
  int v = 0;
  if (cudaStreamSynchronize(stream) != cudaSuccess) return -1;
  if (cudaMemcpyFromSymbol(&v, g_gemm_tc_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // namespace blkq4

extern "C" int blkq4_gemm_plan(int m, int n, int k, size_t workspace_size, int* out6) {
  if (!out6 || m <= 0 || n <= 0 || k <= 0 || (k % 64) != 0) return -1;
  for (int i = 0; i < 6; ++i) out6[i] = 0;
  if (m <= 16) return 0;
  const int sms = blkq4::sm_count() > 0 ? blkq4::sm_count() : 148;
  const blkq4::TcPlan pl = blkq4::plan_tc(m, blkq4::column_tiles(n), blkq4::column_pairs(n), k, workspace_size);
  if (pl.pair) {
    out6[0] = 2; out6[1] = pl.BM; out6[2] = pl.pp.items; out6[3] = 1; out6[4] = pl.pp.balanced;
    out6[5] = pl.pp.balanced ? sms / 2 : 0;
    return 0;
  }
  blkq4::SplitPlan sp = pl.sp;
  const int bm = pl.BM;
  out6[0] = 1; out6[1] = bm; out6[2] = pl.m_tiles * blkq4::column_tiles(n);
  // as many clusters fit of the row-wise kernel as of the column-wise one: one CTA per SM, both
  if (blkq4::have_device())
    blkq4::fit_split(blkq4::choose_kernel<1>(true, bm), out6[2], (k + blkq4::step_k(bm) - 1) / blkq4::step_k(bm), sp);
  out6[3] = sp.split; out6[4] = sp.balanced; out6[5] = sp.balanced ? sms : 0;
  return 0;
}

extern "C" int blkq4_gemm_plan_range_bound(int total_steps, int k_steps, int units, int b) {
  if (total_steps <= 0 || k_steps <= 0 || units <= 0 || b < 0 || b > units) return -1;
  return blkq4::range_bound(total_steps, k_steps, units, b);
}

