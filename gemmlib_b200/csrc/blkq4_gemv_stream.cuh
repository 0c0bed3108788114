// Decode kernel (M <= 8) for column-wise blocks: out[M,N] = A[M,K] x dequant(W4[K,N]).
//
// The weight stream is the only large operand, so the kernel is organised around it.
//
//   * Every warp is its own producer and consumer.  A CTA has eight warps; warp w owns a fixed slice
//     of K (groups of four 64-k steps, the last one of K perhaps shorter: TAIL) of EVERY 16-column tile the CTA works on.  It copies its
//     slice of the packed weights, with the scales and zero points of those steps, into a private
//     ring of shared-memory slots with cp.async (16 bytes per lane, placed as [step][lane], so the
//     later 128-bit reads are conflict free) and waits with cp.async.wait_group, which, unlike a
//     plain load's scoreboard, lets older groups be consumed while younger ones are in flight.
//     D groups per warp are outstanding: 8 warps x 2 groups x 2 KB = 32 KB per CTA, or 64.
//   * Two CTAs fit on an SM and the grid has one CTA per SM (two when the tile count divides well),
//     so with programmatic stream serialization the NEXT launch's CTAs become resident beside this
//     one's, fill their rings, and only then wait for this launch to finish: HBM stays busy across
//     the launches of a decode stack.  Activations are read, and the output written, after that wait.
//   * Math as in the TMA skinny kernel (blkq4_gemv.cu): one packed word becomes four fp16 pairs
//     1024 + q / 64 + q with one shift and four lop3, mma.sync.m16n8k16 takes the weights as its
//     16-row operand and the activations as its 8-column operand, the accumulator of a 64-k step
//     starts at minus the activation-only term of that step, and the step's sum is scaled in fp32:
//         total += scale * (sum_k a_k (magic + q_k) - sum_k a_k (magic + 8)).
//     With zero points zp * sum_k a_k is subtracted from the step's sum, or summed separately, one (step, column) pair per lane
//     (see ZP below).
//   * At the end of a tile the warps leave their partial sums in shared memory, the CTA meets at one
//     barrier, and one warp (rotating) adds them in a fixed order, rounds to fp16 and stores.
//
// Instruction economy matters here: with the copies left out after the first the kernel still takes 0.89 of its time (M = 1,
// 4096 x 11008, B200; 8192 x 28672 0.86), so the ~58 instructions of a 64-k step and their latencies set its pace and not HBM:
// immediate-offset shared-memory loads, no predicates, no index math.
//
// Dequantization numerics: exact in fp32 up to the accumulation order (no fp16 rounding of scale * q);
// equal to the reference kernel's result where that is exact
// (src/mickey/cutlass_ext/q4gemm/warp/quantb_meta_mma_tensor_op_tile_iterator.h:69-104, :436-543).
//
// The instances are spread over three files - blkq4_gemv_stream.cu (one matrix, groups), blkq4_gemv_stream_gather.cu and
// blkq4_gemv_stream_tail.cu - because CUDA loads a file's kernels together when the first of them is launched: with all 92 in one the first
// decode call of a process took 12.4 ms, now 2.5.  Those of the exchange take 128 registers and spill 4 or 8 bytes, the others none.
#pragma once

#include <cstddef>
#include <cstdint>
#include <atomic>
#include <string>

#include "blkq4_common.cuh"
#include "blkq4_stream.cuh"
#include "blkq4_tma.cuh"

namespace blkq4 {
namespace stream {

__device__ __forceinline__ float2 add_f2(const float2& a, const float2& b) { return make_float2(a.x + b.x, a.y + b.y); }
constexpr int kCorrStep = 4 * 16;    // bytes of mma-initialising terms per step: four row pairs, float4 each

// Zero points: none; with sums of their own (up to two rows); subtracted from every step's sum.
enum class Zp { kNone, kOwnSums, kPerStep };

// Quantization blocks as a shift: 2^BS steps of 64 k (blocks of 64 and 128), or 2^-BS blocks in a step (of 32 and 16).
__host__ __device__ constexpr int blocks_per_step(int bs) { return bs < 0 ? 1 << -bs : 1; }
// A ring slot: four steps of weights, a row of 16 scales and one of 16 zero points per block (blocks of 128: per step).
__host__ __device__ constexpr int slot_bytes(int bs) { return kSlotW + kGroupSteps * blocks_per_step(bs) * 48; }
// Halves between the staged activation rows: 16-byte reads of neighbouring rows fall on different banks.
__host__ __device__ constexpr int a_padding(int bs) { return bs < 0 ? 32 : 8; }

struct StreamParams {
  const __half* a;
  __half* out;
  const __half* bias;
  const uint8_t* packed;
  const __half* scales;
  const uint8_t* zp;
  int M, N, K;
  int tiles;        // N / 16
  int steps;        // K / 64
  int a_pitch;      // halves per activation row in shared memory (K + 8: rows land on different banks)
  GemmGroup grp;    // GROUP: the weight matrices whose tiles follow one another; N and the pointers above are unused
  GatherTable gt;   // gather mode: the result goes to every rank's gathered buffer, then to `out` as [M, world * N]
};

constexpr long long kGatherWaitCycles = 2000000000ll;  // ~1 s

// Where an activation is infinite or NaN the accumulators hold NaN: they start at minus the activation-only terms.  One warp puts the
// 16 outputs of such a row right: what they are depends only on the weights of those activations, which are rare, and is found from
// the blocks (of 2^KB k) whose terms in s_corr are not finite.  The weights are those of the other kernels, with two fp16 roundings.
template <int KB, int BLOCK_SHIFT>
__device__ __noinline__ void redo_non_finite_rows(const __half* a, const uint8_t* packed, const __half* scales, const uint8_t* zp, __half* out,
                                                  const __half* bias, int M, int N, int K, const float* s_corr, int tile) {
  const int lane = threadIdx.x & 31, n = tile * 16 + (lane & 15);
  const uint8_t* column = packed + (size_t)(tile * 8 + (lane & 7)) * K + ((lane & 8) ? 1 : 0);
  const int blocks = K >> KB;
  __syncwarp();  // other lanes have stored these outputs
  for (int m = 0; m < M; ++m) {
    float sum = 0.0f;
    bool found = false, all_nan = false;
    for (int b0 = 0; b0 < blocks && !all_nan; b0 += 32) {
      const bool bad = b0 + lane < blocks && !isfinite(s_corr[((size_t)(b0 + lane) * 4 + (m >> 1)) * 4 + (m & 1)]);
      for (uint32_t todo = __ballot_sync(0xffffffffu, bad); todo && !all_nan; todo &= todo - 1) {
        found = true;
        const int first = (b0 + __ffs(todo) - 1) << KB;
        for (int k0 = first; k0 < first + (1 << KB) && !all_nan; k0 += 32) {
          const float own = k0 + lane < first + (1 << KB) ? __half2float(a[(size_t)m * K + k0 + lane]) : 0.0f;
          for (uint32_t ks = __ballot_sync(0xffffffffu, !isfinite(own)); ks && !all_nan; ks &= ks - 1) {
            const int l = __ffs(ks) - 1, k = k0 + l, r = k & 15;
            const float v = __shfl_sync(0xffffffffu, own, l);
            const uint32_t byte = column[(k & ~15) + ((r & 7) >> 1) * 4 + (r & 1) * 2], q = r < 8 ? byte & 15u : byte >> 4;
            const size_t meta = (size_t)(k >> BLOCK_SHIFT) * N + n;
            const __half scale = scales[meta];
            const int z = zp ? (int)zp[meta] : 8;
            sum += v * __half2float(__hfma(scale, __int2half_rn(16 + (int)q), dequant_offset(scale, z)));
            all_nan = __all_sync(0xffffffffu, isnan(sum));
          }
        }
      }
    }
    if (found && lane < 16) {
      const __half h = __float2half_rn(sum);
      out[(size_t)m * N + n] = bias ? __hadd(h, bias[n]) : h;
    }
  }
}

// Shared memory: rings [kWarps][D][slot_bytes] | s_corr [blocks of K, or steps][4] float4 | s_asum [the same][8] (zero points)
//                | s_part [2][PW][16][MS] | s_stage [8][16] fp16 (gather) | s_a [M][a_pitch]
// MZ: rows whose activations are staged at a time: one after the other (2), or all together (8), which saves a round trip to L2 per
// row but runs a longer code.  Two rows one after the other / together, us, block 64 with the early weight fetch: symmetric 512 x 512
// 1.9 / 1.7, 2048 x 1024 2.27 / 2.23, 3072 x 2048 3.5 / 3.3, 4096 x 4096 4.6 / 4.6, 6144 x 4096 5.9 / 5.9 (with zero points 6.4 / 6.4), but
// 6400 x 4096 5.9 / 6.7 (6.4 / 7.4), 7168 x 4096 6.2 / 7.0 (6.6 / 7.5), 8192 x 28672 26.0 / 26.8, 11008 x 4096 8.7 / 9.8: together up to three
// whole groups of steps a warp (6144 k).  With short last groups 6208 x 1024 4.8 / 4.7, 7232 x 2048 5.8 / 5.7: together below 8192 k.
//
// GATHER (N-sharded layer, one process per GPU).  The exchange is latency-bound (a few tens of KB per
// rank), so it carries its own flags: the adding warp stores the tile's results into EVERY rank's
// exchange buffer as 8-byte words {two fp16 results, the call's epoch} - an aligned 8-byte store
// arrives whole, so a word whose flag equals the epoch holds that epoch's data and no fence, counter
// or second flag flight is needed.  When a CTA has finished its tiles it turns receiver: its threads
// poll - bounded - their share of the words of the complete [M, world * N] result in this rank's
// buffer and write the data halves to `out`.  The last CTA advances the rank's epoch.  One launch per
// layer.  Epochs alternate between two buffers: a peer writes epoch e + 2 only after it has received
// this rank's words of epoch e + 1, which this rank sends after its launch of epoch e has completed.
//
// GROUP: several weight matrices of one K read the same activations (the q, k and v projections of a decoder block, or its
// gate and up projections): the tiles of all of them are one sequence, so one launch takes the place of two to four, with
// one ramp, one wait for the preceding launch and one staging of the activations, and its tiles fill the SMs more evenly.
// Measured on B200, graph of two decoder blocks (hidden 4096, 11008; block 64, zero points; 14 layers, 8 launches), M = 1: 102.5 us in
// one launch per layer, 76.5 in groups; M = 4 134.0 / 95.1.
//
// ZP: kPerStep subtracts zp * sum_k a_k from a step's sum before it is scaled, four FMAs and three loads a step.  kOwnSums keeps
// accumulators of their own for these terms, two FMAs and three loads for two steps, but a shuffle, an addition and a store per row
// and 16 more terms per output at the tile's end.  kPerStep is taken for three rows and more.  Measured on B200, kOwnSums / kPerStep,
// us, block 64: M = 8: 2048 x 2048 4.1 / 3.4, 4096 x 4096 7.9 / 6.8, 4096 x 11008 13.5 / 10.8, 8192 x 28672 43.0 / 37.9; M = 4:
// 3.2 / 2.9, 5.9 / 5.5, 10.4 / 9.2, 36.2 / 33.9.  One and two rows keep kOwnSums whatever it costs (M = 1: 512 x 11008 4.3 / 3.5, 4096 x 4096
// 4.4 / 4.2, 4096 x 11008 8.5 / 7.9, 8192 x 28672 27.3 / 28.7): the fp32 sums round otherwise in another order, and a model's results
// would no longer be, to the bit, those it had.  With TAIL it is kPerStep for them too, as the TMA kernel, which had those shapes, has it.
// (As part of the accumulator's initial value, which is a thousand times larger than the sum, the term would be rounded there:
// relative error against 64 bits 2.0853e-4, with either of these 2.0841e-4.)
//
// TAIL: K is not a multiple of 256, or shorter than eight groups of steps.  The steps that are missing from a last group are neither
// copied nor computed; with fewer groups than warps the other warps only take part in the barriers.  The whole groups of other K
// need none of these tests (a kernel of its own: 128 registers already).  Measured on B200 against the TMA kernel, which had
// these shapes (below 512 k the generic kernel), us, symmetric blocks of 128, M = 1, 4 and 8: 256 x 4096 3.4, 3.5, 3.5 / 1.9, 2.3, 3.0;
// 1024 x 4096 3.1, 4.3, 4.5 / 2.2, 2.7, 3.3; 2176 x 8192 5.7, 7.3, 8.3 / 4.2, 5.4, 6.7; 4224 x 11008 10.5, 12.6, 15.2 / 8.6, 10.6, 12.3;
// 3200 x 28672 18.7, 20.1, 23.4 / 12.4, 14.0, 15.4.  Slices balanced to the step, every warp's last group short, were 2 to 9 % slower up
// to 1024 k and equal above: the steps of a short group run one by one.
//
// BS < 0: blocks of 32 and 16, a row of scales and zero points, an activation-only term and a sum per block.  An mma adds up over the
// four lanes of a column, so the lanes share a block's 16-byte chunks: 8 bytes each for blocks of 32, 4 for blocks of 16.  The
// activations are staged in that order, 16 bytes a lane and 32 k, and the chunks lie in the slot so that the reads hit all banks.
// These blocks have the TAIL form only, also where K is whole groups; a form without its tests was not measured.
//
// BS: steps of a quantization block, as a shift (0: blocks of 64, 1: of 128).  The two steps of a 128-k block share scale and
// zero point: one load and conversion of them, two accumulators with independent mma chains, one scaling of their sum.
// (One chain of eight mma from the sum of both activation-only terms is faster still, but the larger partial sums cost
// precision: relative error 2.050e-4 against 2.033e-4 on 8192 k; this 2.033e-4.)  Measured on B200 against a load and scaling per
// step, us: 8192 x 28672 M = 4 28.3 / 28.0, with zero points 36.9 / 36.2, M = 8 33.5 / 32.9; 4096 x 11008, M = 1 7.3 / 7.1.
template <Zp ZP, int D, int MZ, int BS, bool GATHER, bool GROUP, bool TAIL>
__global__ void __launch_bounds__(kWarps * 32, 2)
gemv_stream_kernel(const StreamParams p) {
  extern __shared__ __align__(16) uint8_t s_raw[];
  constexpr int W = kWarps, GS = kGroupSteps;
  constexpr bool HAS_ZP = ZP != Zp::kNone, ZFOLD = ZP == Zp::kPerStep, ZSEP = ZP == Zp::kOwnSums;
  constexpr int PW = ZSEP ? 2 * W : W;  // partial-sum entries per tile: the warps (+ their zero-point terms)
  constexpr int NB = blocks_per_step(BS), kSlotBytes = slot_bytes(BS);
  constexpr int kSlotS = GS * NB * 32;      // scales of a slot: rows of 16 fp16; the zero points, rows of 16 bytes, follow
  const int MS = (p.M + 1) & ~1;
  uint8_t* s_ring = s_raw;
  float* s_corr = reinterpret_cast<float*>(s_ring + W * D * kSlotBytes);
  float* s_asum = s_corr + (size_t)p.steps * NB * 16;
  float* s_part = s_asum + (HAS_ZP ? (size_t)p.steps * NB * 8 : 0);
  __half* s_stage = reinterpret_cast<__half*>(s_part + (size_t)2 * PW * 16 * MS);
  __half* s_a = s_stage + 128;

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int K = p.K, M = p.M;
  int N = p.N;  // GROUP: of the tile that is being loaded
  const int kgroups = (p.steps + GS - 1) / GS;
  // >= 1 without TAIL: the launcher requires kgroups >= W.  Fewer groups than warps go to the first ones, one each (the formula
  // would give them to every second warp, which share two of the SM's four schedulers).
  const bool few = TAIL && kgroups < W;
  const int gb = few ? min(warp, kgroups) : (int)(((long long)kgroups * warp) / W);
  const int myg = few ? (warp < kgroups ? 1 : 0) : (int)(((long long)kgroups * (warp + 1)) / W) - gb;
  const int last_steps = TAIL ? min(GS, p.steps - (gb + myg - 1) * GS) : GS;  // of this warp's last group
  const int my_tiles = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const uint32_t ring_addr = smem_u32(s_ring) + (uint32_t)warp * (D * kSlotBytes);
  const uint32_t ring_last = ring_addr + (D - 1) * kSlotBytes;

  // The next kernel of the stream may become resident now (a no-op unless it was launched with
  // programmatic stream serialization); it fills its rings and then waits for this grid to finish.
  asm volatile("griddepcontrol.launch_dependents;");

  // ---- loader: runs D groups ahead of the consumer; all addresses advance incrementally ----
  const long long w_tile_adj = (long long)gridDim.x * 8 * K - (long long)myg * (GS * 64);
  // The first 2 R lanes copy the scales of row lane / 2 (blocks of 64: of a step), column half lane % 2, the next R the zero points
  // of row lane - 2 R; with blocks of 16 (R = 16) the zero points take a copy of their own by lanes 0 to 15.
  constexpr int R = GS * NB;
  constexpr bool kZpApart = 3 * R > 32;
  const int zp_row = BS >= 0 ? (lane - 2 * GS) % GS : lane % R;  // (2 R is a multiple of R)
  const uint32_t meta_lane = (lane < 2 * R || (HAS_ZP && lane < 3 * R)) ? 1u : 0u;
  const uint32_t z_dst = kSlotW + kSlotS + zp_row * 16;
  const uint32_t m_dst = lane < 2 * R ? kSlotW + (lane >> 1) * 32 + (lane & 1) * 16 : z_dst;
  const int meta_step = lane < 2 * R ? (lane >> 1) / NB : zp_row / NB;  // step whose scales / zero points this lane copies
  // A weight chunk's place in the slot: chunk t of packed column g at 4 g + t, in another order where lanes read 8 or 4 of its
  // 16 bytes (blocks of 32 and 16), so that they fall on different banks.
  const int chunk_xor = BS == -1 ? (g & 2) : BS == -2 ? (g >> 1) & 3 : 0;
  const uint32_t w_dst = (uint32_t)(BS >= 0 ? lane : 4 * g + (t ^ chunk_xor)) * 16u;
  const uint8_t *wp, *mp, *zq = nullptr;  // zq: kZpApart
  long long z_step = 0, z_tile_adj = 0;
  long long m_step, m_tile_adj;
  // this lane's addresses for the warp's first group of a tile
  auto point_at = [&](const uint8_t* packed, const __half* scales, const uint8_t* zp, int tile) {
    wp = packed + (size_t)(tile * 8 + g) * K + (size_t)gb * (GS * 64) + t * 16;
    constexpr int rows_per_group = BS > 0 ? GS >> BS : R;
    auto row_of = [&](int r) { return BS > 0 ? (gb * GS + r) >> BS : gb * R + r; };  // r: of the slot; blocks of 128 have theirs twice
    if (lane < 2 * R) {
      const int r = lane >> 1, h = lane & 1;
      mp = reinterpret_cast<const uint8_t*>(scales) + ((size_t)row_of(r) * N + tile * 16 + h * 8) * 2;
      m_step = (long long)rows_per_group * N * 2;
      m_tile_adj = (long long)gridDim.x * 32 - (long long)myg * m_step;
    } else {
      mp = (HAS_ZP ? zp : packed) + (size_t)row_of(zp_row) * N + tile * 16;  // only used with zero points
      m_step = (long long)rows_per_group * N;
      m_tile_adj = (long long)gridDim.x * 16 - (long long)myg * m_step;
    }
    if (HAS_ZP && kZpApart) {
      zq = zp + (size_t)row_of(zp_row) * N + tile * 16;
      z_step = (long long)rows_per_group * N;
      z_tile_adj = (long long)gridDim.x * 16 - (long long)myg * z_step;
    }
  };
  int ld_tile = blockIdx.x;
  if constexpr (GROUP) {
    const int i = p.grp.of_tile(ld_tile);
    N = p.grp.n[i];
    point_at(p.grp.packed[i], p.grp.scales[i], p.grp.zp[i], ld_tile - p.grp.first_tile(i));
  } else {
    point_at(p.packed, p.scales, p.zp, ld_tile);
  }
  int ld_left = my_tiles * myg, ld_j = 0;
  auto issue_group = [&](uint32_t dst) {
    const uint32_t go = ld_left > 0 ? 1u : 0u;
    const uint32_t dw = dst + w_dst;
    if constexpr (TAIL) {
      // steps past the end of K are neither copied nor computed
      const int n = go ? (ld_j + 1 == myg ? last_steps : GS) : 0;
      cp_async16_if<0>(dw, wp, n > 0);
      cp_async16_if<64>(dw, wp, n > 1);
      cp_async16_if<128>(dw, wp, n > 2);
      cp_async16_if<192>(dw, wp, n > 3);
      cp_async16_if<0>(dst + m_dst, mp, meta_lane && meta_step < n);
      if (HAS_ZP && kZpApart) cp_async16_if<0>(dst + z_dst, zq, lane < R && zp_row / NB < n);
    } else {
      cp_async16_if<0>(dw, wp, go);
      cp_async16_if<64>(dw, wp, go);
      cp_async16_if<128>(dw, wp, go);
      cp_async16_if<192>(dw, wp, go);
      cp_async16_if<0>(dst + m_dst, mp, go & meta_lane);
      static_assert(!kZpApart, "blocks of 16: TAIL");
    }
    cp_async_commit();  // always: the group count per iteration stays fixed
    --ld_left;
    const bool wrap = ++ld_j == myg;
    if constexpr (GROUP) {
      wp += GS * 64;
      mp += m_step;
      if (wrap) {
        ld_j = 0;
        ld_tile += (int)gridDim.x;
        if (ld_tile < p.tiles) {
          const int i = p.grp.of_tile(ld_tile);
          N = p.grp.n[i];
          point_at(p.grp.packed[i], p.grp.scales[i], p.grp.zp[i], ld_tile - p.grp.first_tile(i));
        }
      }
    } else {
      wp += (GS * 64) + (wrap ? w_tile_adj : 0);
      mp += m_step + (wrap ? m_tile_adj : 0);
      if (HAS_ZP && kZpApart) zq += z_step + (wrap ? z_tile_adj : 0);
      if (wrap) ld_j = 0;
    }
  };
  // Weights, scales and zero points are read WITHOUT waiting for the preceding kernel of the stream
  // (the caller vouches for them when it asks for the early start).
  {
    uint32_t dst = ring_addr;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      issue_group(dst);
      dst += kSlotBytes;
    }
  }

  // Activations and the output belong to stream order.
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // Gather mode: this call's epoch is one past the calls this rank has completed (the word changes
  // only at the very end of a launch, and the preceding launch has completed: see the wait above).
  unsigned gather_epoch = 0;
  size_t gather_off = 0;
  if (GATHER) {
    gather_epoch = *reinterpret_cast<volatile unsigned*>(p.gt.base[p.gt.rank] + kGatherEpochOff) + 1u;
    gather_off = kGatherCtrlBytes + (size_t)(2 + 2 * (gather_epoch & 1u)) * p.gt.buf_bytes;  // flagged-word buffers follow the two fp16 ones
  }

  // ---- per warp: its own K slice of the activations into shared memory, and the activation-only
  //      terms of its steps.  Chunk c = 8 halves; even c is the "lo" half (k % 16 < 8) of a 16-k block.
  //      symmetric:   term = -(1024 lo + 64 hi + 8 (lo + hi));   zero points: -(1024 lo + 64 hi) and lo + hi
  {
    const int slice_k0 = gb * (GS * 64);
    const int chunks = myg * (GS * 8);  // a multiple of 32
    // TAIL: lanes past the end of K run along (the shuffles below are of whole warps) with zeros and store nothing
    auto load_chunk = [&](int m, int k0) {
      if (TAIL && k0 >= K) return make_uint4(0u, 0u, 0u, 0u);
      return __ldg(reinterpret_cast<const uint4*>(p.a + (size_t)m * K + k0));
    };
    auto finish_row = [&](int m, int k0, const uint4& v) {
      if (!TAIL || k0 < K) {
        if constexpr (BS >= 0) {
          *reinterpret_cast<uint4*>(s_a + (size_t)m * p.a_pitch + k0) = v;
        } else {
          // per 32 k, lane t's 16 bytes: of its chunk the k of its two words (blocks of 32: k, then k + 8), or of both chunks
          // those of its word (blocks of 16)
          uint8_t* d = reinterpret_cast<uint8_t*>(s_a + (size_t)m * p.a_pitch + (k0 & ~31));
          const int cb = (k0 >> 4) & 1, hi = (k0 >> 3) & 1;
          if constexpr (BS == -1) {
            *reinterpret_cast<uint2*>(d + 32 * cb + 8 * hi) = make_uint2(v.x, v.y);
            *reinterpret_cast<uint2*>(d + 32 * cb + 16 + 8 * hi) = make_uint2(v.z, v.w);
          } else {
            uint32_t* q = reinterpret_cast<uint32_t*>(d + 8 * cb + 4 * hi);
            q[0] = v.x; q[4] = v.y; q[8] = v.z; q[12] = v.w;
          }
        }
      }
      const __half2* h = reinterpret_cast<const __half2*>(&v);
      float s = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(h[e]);
        s += f.x + f.y;
      }
      // the lanes of a block (eight of a step, for blocks of 64): sum the chunks of equal parity, then pair lo with hi
      if (BS >= -1) s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (BS >= 0) s += __shfl_xor_sync(0xffffffffu, s, 4);
      const float other = __shfl_xor_sync(0xffffffffu, s, 1);
      if ((lane & (8 / NB - 1)) == 0 && (!TAIL || k0 < K)) {
        const float lo = s, hi = other;
        const int step = k0 >> (BS < 0 ? 6 + BS : 6);  // a block where a step holds several
        // one float4 per row pair (m even, m odd, m even, m odd): the accumulator rows n and n + 8 start alike
        float* dst = s_corr + ((size_t)step * 4 + (m >> 1)) * 4 + (m & 1);
        const float nb = -(1024.0f * lo + 64.0f * hi);
        const float c = HAS_ZP ? nb : nb - 8.0f * (lo + hi);
        dst[0] = c;
        dst[2] = c;
        if (HAS_ZP) s_asum[(size_t)step * 8 + m] = lo + hi;
      }
    };
    if (MZ == 2) {
      for (int m = 0; m < M; ++m)
        for (int c0 = 0; c0 < chunks; c0 += 32) {
          const int k0 = slice_k0 + (c0 + lane) * 8;
          finish_row(m, k0, load_chunk(m, k0));
        }
    } else {
      // several rows: all rows' loads of a chunk first (one L2 round trip per chunk, not one per row)
      for (int c0 = 0; c0 < chunks; c0 += 32) {
        const int k0 = slice_k0 + (c0 + lane) * 8;
        uint4 v[8];
#pragma unroll
        for (int m = 0; m < 8; ++m)
          if (m < M) v[m] = load_chunk(m, k0);
#pragma unroll
        for (int m = 0; m < 8; ++m)
          if (m < M) finish_row(m, k0, v[m]);
      }
    }
  }
  __syncwarp();

  constexpr uint32_t kLoMask = 0x000f000fu, kHiMask = 0x00f000f0u;
  constexpr uint32_t kLoMagic = 0x64006400u, kHiMagic = 0x54005400u;
  // rows >= M of the activation operand repeat row M - 1; their outputs are never stored
  const uint32_t a_base = smem_u32(s_a) + (uint32_t)(min(g, M - 1) * p.a_pitch + gb * (GS * 64) + t * (BS < 0 ? 8 : 16)) * 2u;
  const uint32_t c_base = smem_u32(s_corr) + (uint32_t)(gb * R) * kCorrStep + (uint32_t)t * 16u;
  const uint32_t asum_base = smem_u32(s_asum) + (uint32_t)(gb * R) * 32u;

  float total[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  float ztot[2] = {0.0f, 0.0f};  // ZSEP: zero-point terms of column (lane & 15), rows m, over the steps of half (lane >> 4)

  // where in a slot this lane's weights of a step's blocks lie (BS < 0)
  uint32_t w_at[NB];
#pragma unroll
  for (int b = 0; BS < 0 && b < NB; ++b)
    w_at[b] = BS == -1 ? (uint32_t)((4 * g + ((2 * b + (t >> 1)) ^ chunk_xor)) * 16 + (t & 1) * 8)
                       : (uint32_t)((4 * g + (b ^ chunk_xor)) * 16 + t * 4);

  uint32_t src = ring_addr;
  float zeros = 0.0f;  // TAIL: NaN once this lane has added up an output that is
  // The warps look at it once, after their last tile.  (A vote per tile takes up to a tenth where a CTA has many short tiles; but the
  // compiler's schedule of the steps of symmetric blocks of 128 is better with it: M = 1, 2 and 4 1.03, 1.00 and 0.99 of the time without
  // either, at the end 1.05, 1.03 and 1.03.)
  constexpr bool kVotePerTile = TAIL && BS == 1 && ZP == Zp::kNone;
  auto redo_tile = [&](int tl) {
    redo_non_finite_rows<(BS < 0 ? 6 + BS : 6), 6 + BS>(p.a, p.packed, p.scales, p.zp, p.out, p.bias, M, N, K, s_corr, blockIdx.x + tl * gridDim.x);
  };
  for (int tl = 0; tl < my_tiles; ++tl) {
    uint32_t a_addr = a_base, c_addr = c_base, as_addr = asum_base;
    for (int j2 = 0; j2 < myg; ++j2) {
      cp_async_wait<D - 1>();
      __syncwarp();  // the scales / zero points of the slot were copied by other lanes
      const uint32_t src_w = src + lane * 16;
      const uint32_t src_s = src + kSlotW + g * 2;
      const int n_steps = TAIL && j2 + 1 == myg ? last_steps : GS;
      const uint32_t src_z = src + kSlotW + kSlotS + g, as_t = as_addr + t * 8;
      if (ZSEP) {
        const uint32_t col = lane & 15, u0 = (lane >> 4) * (GS / 2);
#pragma unroll
        for (int uu = 0; uu < GS / 2; uu += 1 << BS) {
          const uint32_t u = u0 + uu;
          if (TAIL && (int)u >= n_steps) break;
          const float s = lds_half_as_float<0>(src + kSlotW + u * 32 + col * 2);
          const float z = lds_u8_as_float(src + kSlotW + kSlotS + u * 16 + col);
          const float nsz = -s * z;
#pragma unroll
          for (int v = 0; v < (1 << BS); ++v) {
            // Always.  Without the branch nvcc 12.9 schedules blocks of 128 up to 2 % slower (M = 1 4096 x 11008 7.9 / 8.0, 8192 x 28672 26.1 /
            // 26.7 us; blocks of 64 alike): to be timed again with another compiler.
            if (M > 0) {
              const float2 as = lds_f2<0>(as_addr + (u + v) * 32);
              ztot[0] = fmaf(nsz, as.x, ztot[0]);
              ztot[1] = fmaf(nsz, as.y, ztot[1]);
            }
          }
        }
      }
#define BLKQ4_STREAM_UNPACK(U)                                                                  \
        const uint4 wv##U = lds_v4<(U) * 512>(src_w);                                           \
        const uint4 v0##U = lds_v4<(U) * 128>(a_addr), v1##U = lds_v4<(U) * 128 + 16>(a_addr);  \
        uint32_t lo_a##U[4], lo_b##U[4], hi_a##U[4], hi_b##U[4];                                \
        const uint32_t w4##U[4] = {wv##U.x, wv##U.y, wv##U.z, wv##U.w};                         \
        _Pragma("unroll") for (int r = 0; r < 4; ++r) {                                         \
          const uint32_t x = w4##U[r], y = x >> 8;                                              \
          lo_a##U[r] = lop3_and_or(x, kLoMask, kLoMagic); /* (n;     k 2r, 2r+1)   1024 + q */  \
          hi_a##U[r] = lop3_and_or(x, kHiMask, kHiMagic); /* (n;     k 2r+8, 2r+9)   64 + q */  \
          lo_b##U[r] = lop3_and_or(y, kLoMask, kLoMagic); /* (n + 8; k 2r, 2r+1)            */  \
          hi_b##U[r] = lop3_and_or(y, kHiMask, kHiMagic); /* (n + 8; k 2r+8, 2r+9)          */  \
        }
#define BLKQ4_STREAM_ZP(U, ACC, AS)                                                             \
        {                                                                                       \
          const float za = lds_u8_by_mantissa<(U) * 16>(src_z), zb = lds_u8_by_mantissa<(U) * 16 + 8>(src_z); \
          const float2 as = AS;                                                                 \
          ACC[0] = fmaf(-za, as.x, ACC[0]);                                                     \
          ACC[1] = fmaf(-za, as.y, ACC[1]);                                                     \
          ACC[2] = fmaf(-zb, as.x, ACC[2]);                                                     \
          ACC[3] = fmaf(-zb, as.y, ACC[3]);                                                     \
        }
#define BLKQ4_STREAM_MMA(U)                                                                     \
        float acc##U[4];                                                                        \
        {                                                                                       \
          const float4 c = lds_f4<(U) * kCorrStep>(c_addr);                                     \
          mma_init(acc##U, lo_a##U[0], lo_b##U[0], lo_a##U[1], lo_b##U[1], v0##U.x, v0##U.y, c); \
        }                                                                                       \
        mma_acc(acc##U, lo_a##U[2], lo_b##U[2], lo_a##U[3], lo_b##U[3], v0##U.z, v0##U.w);      \
        mma_acc(acc##U, hi_a##U[0], hi_b##U[0], hi_a##U[1], hi_b##U[1], v1##U.x, v1##U.y);      \
        mma_acc(acc##U, hi_a##U[2], hi_b##U[2], hi_a##U[3], hi_b##U[3], v1##U.z, v1##U.w);
#define BLKQ4_STREAM_SCALE(U, X0, X1, X2, X3)                                                   \
        /* accumulator rows n (e = 0, 1) and n + 8 (e = 2, 3); columns m = 2 t + (e & 1) */     \
        const float sa = lds_half_as_float<(U) * 32>(src_s);                                    \
        const float sb = lds_half_as_float<(U) * 32 + 16>(src_s);                               \
        total[0] = fmaf(sa, X0, total[0]);                                                      \
        total[1] = fmaf(sa, X1, total[1]);                                                      \
        total[2] = fmaf(sb, X2, total[2]);                                                      \
        total[3] = fmaf(sb, X3, total[3]);
#define BLKQ4_STREAM_STEP(U)                                                                    \
      {                                                                                         \
        BLKQ4_STREAM_UNPACK(U)                                                                  \
        BLKQ4_STREAM_MMA(U)                                                                     \
        if (ZFOLD) BLKQ4_STREAM_ZP(U, acc##U, lds_f2<(U) * 32>(as_t))                           \
        BLKQ4_STREAM_SCALE(U, acc##U[0], acc##U[1], acc##U[2], acc##U[3])                       \
      }
#define BLKQ4_STREAM_BLOCK128(U, V)                                                             \
      {                                                                                         \
        BLKQ4_STREAM_UNPACK(U)                                                                  \
        BLKQ4_STREAM_UNPACK(V)                                                                  \
        BLKQ4_STREAM_MMA(U)                                                                     \
        BLKQ4_STREAM_MMA(V)                                                                     \
        float sum[4];                                                                           \
        _Pragma("unroll") for (int e = 0; e < 4; ++e) sum[e] = acc##U[e] + acc##V[e];           \
        if (ZFOLD) BLKQ4_STREAM_ZP(U, sum, add_f2(lds_f2<(U) * 32>(as_t), lds_f2<(V) * 32>(as_t))) \
        BLKQ4_STREAM_SCALE(U, sum[0], sum[1], sum[2], sum[3])                                   \
      }
/* Blocks of 32: block J of step U; 8 bytes of weights, two words, per lane. */
#define BLKQ4_STREAM_BLOCK32(U, J)                                                              \
      {                                                                                         \
        const uint2 w = lds_v2<(U) * 512>(src + w_at[J]);                                       \
        const uint4 v = lds_v4<(U) * 128 + (J) * 64>(a_addr);                                   \
        const uint32_t y0 = w.x >> 8, y1 = w.y >> 8;                                            \
        float acc[4];                                                                           \
        const float4 c = lds_f4<((U) * NB + (J)) * kCorrStep>(c_addr);                          \
        mma_init(acc, lop3_and_or(w.x, kLoMask, kLoMagic), lop3_and_or(y0, kLoMask, kLoMagic),  \
                 lop3_and_or(w.y, kLoMask, kLoMagic), lop3_and_or(y1, kLoMask, kLoMagic), v.x, v.y, c); \
        mma_acc(acc, lop3_and_or(w.x, kHiMask, kHiMagic), lop3_and_or(y0, kHiMask, kHiMagic),   \
                lop3_and_or(w.y, kHiMask, kHiMagic), lop3_and_or(y1, kHiMask, kHiMagic), v.z, v.w); \
        if (ZFOLD) BLKQ4_STREAM_ZP((U) * NB + (J), acc, lds_f2<((U) * NB + (J)) * 32>(as_t))    \
        BLKQ4_STREAM_SCALE((U) * NB + (J), acc[0], acc[1], acc[2], acc[3])                      \
      }
/* Blocks of 16: block C of step U; one word per lane.  V: activations of its block pair. */
#define BLKQ4_STREAM_BLOCK16(U, C, V0, V1)                                                      \
      {                                                                                         \
        const uint32_t x = lds_u32<(U) * 512>(src + w_at[C]), y = x >> 8;                       \
        float acc[4];                                                                           \
        const float4 c = lds_f4<((U) * NB + (C)) * kCorrStep>(c_addr);                          \
        mma_init(acc, lop3_and_or(x, kLoMask, kLoMagic), lop3_and_or(y, kLoMask, kLoMagic),     \
                 lop3_and_or(x, kHiMask, kHiMagic), lop3_and_or(y, kHiMask, kHiMagic), V0, V1, c); \
        if (ZFOLD) BLKQ4_STREAM_ZP((U) * NB + (C), acc, lds_f2<((U) * NB + (C)) * 32>(as_t))    \
        BLKQ4_STREAM_SCALE((U) * NB + (C), acc[0], acc[1], acc[2], acc[3])                      \
      }
#define BLKQ4_STREAM_SMALL(U)                                                                   \
      {                                                                                         \
        if constexpr (BS == -1) {                                                               \
          BLKQ4_STREAM_BLOCK32(U, 0)                                                            \
          BLKQ4_STREAM_BLOCK32(U, 1)                                                            \
        } else {                                                                                \
          const uint4 p0 = lds_v4<(U) * 128>(a_addr), p1 = lds_v4<(U) * 128 + 64>(a_addr);      \
          BLKQ4_STREAM_BLOCK16(U, 0, p0.x, p0.y)                                                \
          BLKQ4_STREAM_BLOCK16(U, 1, p0.z, p0.w)                                                \
          BLKQ4_STREAM_BLOCK16(U, 2, p1.x, p1.y)                                                \
          BLKQ4_STREAM_BLOCK16(U, 3, p1.z, p1.w)                                                \
        }                                                                                       \
      }
      if constexpr (BS < 0) {
        BLKQ4_STREAM_SMALL(0)
        if (n_steps > 1) BLKQ4_STREAM_SMALL(1)
        if (n_steps > 2) BLKQ4_STREAM_SMALL(2)
        if (n_steps > 3) BLKQ4_STREAM_SMALL(3)
      } else if constexpr (BS == 1) {
        BLKQ4_STREAM_BLOCK128(0, 1)
        if (n_steps > 2) BLKQ4_STREAM_BLOCK128(2, 3)  // K is a whole number of blocks
      } else if (n_steps == GS) {
        BLKQ4_STREAM_STEP(0)
        BLKQ4_STREAM_STEP(1)
        BLKQ4_STREAM_STEP(2)
        BLKQ4_STREAM_STEP(3)
      } else {
        BLKQ4_STREAM_STEP(0)
        if (n_steps > 1) BLKQ4_STREAM_STEP(1)
        if (n_steps > 2) BLKQ4_STREAM_STEP(2)
      }
#undef BLKQ4_STREAM_SMALL
#undef BLKQ4_STREAM_BLOCK16
#undef BLKQ4_STREAM_BLOCK32
#undef BLKQ4_STREAM_BLOCK128
#undef BLKQ4_STREAM_STEP
#undef BLKQ4_STREAM_SCALE
#undef BLKQ4_STREAM_MMA
#undef BLKQ4_STREAM_ZP
#undef BLKQ4_STREAM_UNPACK
      issue_group(src);  // refill the slot just consumed
      src = (src == ring_last) ? ring_addr : src + kSlotBytes;
      a_addr += GS * 128;
      c_addr += R * kCorrStep;
      as_addr += R * 32;
    }
    // ---- tile end: double-buffered partial sums, one CTA barrier, one warp (rotating) adds them up.
    //      The adder of tile tl reaches the barrier of tile tl + 1 only after it has read the buffer,
    //      and nobody writes that buffer again before the barrier of tile tl + 1. ----
    float* buf = s_part + (size_t)(tl & 1) * (PW * 16 * MS);
    if (2 * t < M) {
      float* d0 = buf + ((size_t)warp * 16 + g) * MS + 2 * t;
      *reinterpret_cast<float2*>(d0) = make_float2(total[0], total[1]);
      *reinterpret_cast<float2*>(d0 + 8 * MS) = make_float2(total[2], total[3]);
    }
    total[0] = total[1] = total[2] = total[3] = 0.0f;
    if (ZSEP) {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        if (m < MS) {
          const float z = ztot[m] + __shfl_xor_sync(0xffffffffu, ztot[m], 16);
          if (lane < 16) buf[((size_t)(W + warp) * 16 + lane) * MS + m] = z;
          ztot[m] = 0.0f;
        }
      }
    }
    __syncthreads();
    if (warp == tl % W) {
      int tile = blockIdx.x + tl * gridDim.x, n_out = p.N;
      __half* out = p.out;
      const __half* bias = p.bias;
      if constexpr (GROUP) {
        const int i = p.grp.of_tile(tile);
        tile -= p.grp.first_tile(i);
        n_out = p.grp.n[i];
        out = p.grp.out[i];
        bias = p.grp.bias[i];
      }
      for (int idx = lane; idx < 16 * M; idx += 32) {
        const int row = idx & 15, m = idx >> 4;
        float sum = 0.0f;
#pragma unroll
        for (int w2 = 0; w2 < PW; ++w2) sum += buf[((size_t)w2 * 16 + row) * MS + m];
        const int n = tile * 16 + row;
        // bias joins the ROUNDED result in fp16, as a separate `output += bias` would
        const __half h = __float2half_rn(sum);
        if (GATHER) s_stage[idx] = h;  // [m][16]
        else out[(size_t)m * n_out + n] = bias ? __hadd(h, bias[n]) : h;
        if (TAIL) zeros = fmaf(sum, 0.0f, zeros);
      }
      if (kVotePerTile) {
        if (__any_sync(0xffffffffu, isnan(zeros))) redo_tile(tl);
        zeros = 0.0f;
      }
      if (GATHER) {
        // this rank's 16 columns of row m as eight flagged words, into every rank's buffer
        __syncwarp();
        for (int w = lane; w < 8 * M; w += 32) {
          const int m = w >> 3, pair = w & 7;
          const uint32_t data = *reinterpret_cast<const uint32_t*>(s_stage + m * 16 + pair * 2);
          const size_t word = ((size_t)m * p.gt.n_total + (size_t)p.gt.rank * N + (size_t)tile * 16) / 2 + pair;
          for (int r = 0; r < p.gt.world; ++r) st_relaxed_sys_v2(p.gt.base[r] + gather_off + word * 8, data, gather_epoch);
        }
        __syncwarp();
      }
    }
  }
  cp_async_wait<0>();
  if (TAIL && !kVotePerTile && __any_sync(0xffffffffu, isnan(zeros)))
    for (int tl = warp; tl < my_tiles; tl += W) redo_tile(tl);  // the tiles that this warp has added up
  if (GATHER) {
    uint8_t* local = p.gt.base[p.gt.rank];
    // receiver: this CTA's share of the words of the complete result
    const unsigned long long nwords = (unsigned long long)M * p.gt.n_total / 2;
    const uint8_t* src = local + gather_off;
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.out);
    bool expired = false;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < nwords;
         i += (unsigned long long)gridDim.x * blockDim.x) {
      uint2 w = ld_relaxed_sys_v2(src + i * 8);
      if (w.y != gather_epoch && !expired) {
        const long long t0 = clock64();
        while ((w = ld_relaxed_sys_v2(src + i * 8)).y != gather_epoch) {
          if (clock64() - t0 > kGatherWaitCycles) {
            // which rank's columns are missing: word i covers columns 2 (i % (n_total / 2)), + 1
            const int col = (int)(i % (unsigned long long)(p.gt.n_total / 2)) * 2;
            atomicCAS(reinterpret_cast<int*>(local + kGatherErrorOff), 0, 0x400 | (col / N));
            expired = true;  // this thread stops waiting for its other words too
            break;
          }
        }
      }
      if (w.y == gather_epoch) dst[i] = w.x;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned arrived = atomicAdd(reinterpret_cast<unsigned*>(local + kGatherDoneOff), 1u);
      if (arrived == gridDim.x - 1) {
        // last CTA of this rank: keep the two-kernel protocol's ticket numbering in step (its wait
        // kernel draws kGatherWaitCtas tickets per call) and advance the epoch
        *reinterpret_cast<volatile unsigned*>(local + kGatherDoneOff) = 0u;
        atomicAdd(reinterpret_cast<unsigned*>(local + kGatherTicketOff), (unsigned)kGatherWaitCtas);
        __threadfence();
        *reinterpret_cast<volatile unsigned*>(local + kGatherEpochOff) = gather_epoch;
      }
    }
  }
}

struct StreamLaunch {
  StreamParams p;
  size_t smem;
  int grid, ring;    // groups per ring: 2 or 4
  bool one_by_one;   // MZ = 2
  Zp zp;
  cudaStream_t stream;
  bool early;
};

template <Zp ZP, int D, int MZ, int BS, bool GATHER, bool GROUP, bool TAIL>
std::string launch_instance(const StreamLaunch& l) {
  auto kern = gemv_stream_kernel<ZP, D, MZ, BS, GATHER, GROUP, TAIL>;
  static std::atomic<int> granted[64];
  cudaError_t e = ensure_dynamic_smem(kern, l.smem, granted);
  if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(l.grid);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = l.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = l.early ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kern, l.p);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
  return std::string();
}

template <Zp ZP, int BS, bool GATHER, bool GROUP, bool TAIL>
std::string launch_zp(const StreamLaunch& l) {
  if constexpr (ZP != Zp::kPerStep || TAIL)  // else three rows and more
    if (l.one_by_one)
      return l.ring == 4 ? launch_instance<ZP, 4, 2, BS, GATHER, GROUP, TAIL>(l) : launch_instance<ZP, 2, 2, BS, GATHER, GROUP, TAIL>(l);
  return l.ring == 4 ? launch_instance<ZP, 4, 8, BS, GATHER, GROUP, TAIL>(l) : launch_instance<ZP, 2, 8, BS, GATHER, GROUP, TAIL>(l);
}

template <int BS, bool GATHER, bool GROUP, bool TAIL>
std::string launch_stream(const StreamLaunch& l) {
  if (l.zp == Zp::kNone) return launch_zp<Zp::kNone, BS, GATHER, GROUP, TAIL>(l);
  if constexpr (!TAIL)
    if (l.zp == Zp::kOwnSums) return launch_zp<Zp::kOwnSums, BS, GATHER, GROUP, TAIL>(l);
  return launch_zp<Zp::kPerStep, BS, GATHER, GROUP, TAIL>(l);
}

// bs: see BS
std::string launch_stream_gather(int bs, const StreamLaunch& l);
std::string launch_stream_tail(int bs, const StreamLaunch& l);

}  // namespace stream
}  // namespace blkq4
