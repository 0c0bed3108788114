// Tensor-core kernel for a few rows (M <= 16) and column-wise blocks of 64 or 128: out[M,N] = A[M,K] x dequant(W4[K,N]).
//
// The TMA -> dequantizer -> tensor memory -> tcgen05.mma pipeline of blkq4_gemm_tc.cu, with the other skinny kernels' numerics:
// the weights are multiplied as the integers q - zp, which fp16 holds exactly, and every quantization block's sum is scaled in fp32.
// A block therefore has an accumulator of its own (16 columns of tensor memory, a ring of eight), which four warps read a step
// at a time, scale and add up in registers while the next steps are multiplied:
//
//   D_b^T[128 n x 16 m] (TMEM, fp32)  =  (q - zp)^T[128 n x block k] (TMEM, fp16)  x  A[16 m x block k]^T (smem)
//   total[m] (registers)  +=  scale[b][n] * D_b[n][m]
//
// Measured on B200 against those kernels (TMA and wide skinny kernels), M = 16, block 64 with zero points (block 128 symmetric), us:
// 512 x 512 4.0 / 2.5 (3.9 / 2.4); 1024 x 4096 5.8 / 3.8 (4.7 / 3.6); 4096 x 4096 10.8 / 6.9 (10.3 / 6.5); 4096 x 11008 21.5 / 12.8
// (20.5 / 11.9); 11008 x 4096 26.5 / 11.8 (25.2 / 10.9); 8192 x 28672 85.6 / 45.1 (73.4 / 42.0); 1024 x 28672 19.0 / 7.9 (18.3 / 7.3).
// Relative error against 64 bits 2.08e-4 (2.10e-4 there).
//
// What bounds it: as in blkq4_gemm_tc.cu up to 64 rows the dequantizers' instructions, five for four weights (a shift, two
// lop3, two subtractions) where the scaled fp16 weights take six, and the 16 multiply-adds of a block, eight packed ones.
// The activations of 16 rows are read once per tile of 128 columns; the kernels that had these shapes read them once per 16 or 32
// columns (from L2: 256 KB at K = 8192).
//
// A CTA takes whole tiles in turn, or a part of the K of one tile, whose CTAs form a cluster and exchange their fp32 sums through
// distributed shared memory, added in part order.
//
// Warp roles: 0 to 3 scale and store; then kGroups groups of four dequantizer warps, on steps of 128 k in turn; three TMA
// producers (activations; packed weights; scales and zero points); last the MMA issuer.
#include <cstddef>
#include <cstdint>
#include <atomic>
#include <string>

#include "blkq4_common.cuh"
#include "blkq4_tc.cuh"
#include "blkq4_tma.cuh"
#include "ms_blkq4gemm.h"

namespace blkq4 {

__device__ int g_skinny_tc_error = 0;  // 0 ok; otherwise (role << 8) | barrier id of the wait that gave up

namespace {

using namespace tc;

constexpr int kRows = 16;           // activation rows of a tile = UMMA N
constexpr int kSub = 2, kStepK = kSub * BLOCK_K;  // a step: 128 k
constexpr int kRing = 6;            // stages of activations and of dequantized weights (64 TMEM columns each)
constexpr int kStages = 12;         // stages of packed weights, scales and zero points
constexpr int kAccCols = 128;       // tensor memory of the accumulators: one of 16 columns per quantization block of a step
constexpr int kMaxAccs = 8;         // steps whose sums fit there: eight of one block, four of two
constexpr int kGroups = 2;          // dequantizer groups: with three or four a launch starts later, and only 8192 x 28672 gains (1 %).
                                    // Two / three / four, us, M = 16: 512 x 512 2.5 / 2.8 / 2.9; 4096 x 4096 6.9 / 7.0 / 7.3;
                                    // 4096 x 11008 12.8 / 12.9 / 13.8; one: 2.5, 7.3, 14.7
constexpr int kFirstDeqWarp = 4, kActWarp = kFirstDeqWarp + 4 * kGroups, kWeightWarp = kActWarp + 1, kMetaWarp = kActWarp + 2,
              kMmaWarp = kActWarp + 3, kThreads = 32 * (kMmaWarp + 1);
constexpr int kActBytes = kSub * kRows * 128, kPackBytes = kSub * kPackTileBytes, kScaleBytes = kSub * TILE_N * 2, kZpBytes = kSub * TILE_N;
constexpr uint32_t kDeqCol0 = kAccCols, kTmemCols = 512;
static_assert(kDeqCol0 + kRing * kSub * kDeqCols <= kTmemCols);
constexpr int kMaxSplit = 8;
static_assert(kMaxSplit * TILE_N * 16 <= kRing * kActBytes, "the exchange of a split lies over the activation ring");

constexpr uint32_t kActOff = 0, kPackOff = kActOff + kRing * kActBytes, kScaleOff = kPackOff + kStages * kPackBytes,
                   kZpOff = kScaleOff + kStages * kScaleBytes, kBarOff = kZpOff + kStages * kZpBytes, kSmemBytes = kBarOff + 512 + 1024;

enum : int {
  kFull = 0,                       // [kStages] packed weights and meta landed
  kPackFree = kFull + kStages,     // [kStages] read by the dequantizers, and the scales by the adders
  kStepFull = kPackFree + kStages, // [kRing] operands of the step are there
  kMmaDone = kStepFull + kRing,    // [kRing] its MMAs have retired
  kAccFull = kMmaDone + kRing,     // [kMaxAccs] the sums of a step are complete
  kAccEmpty = kAccFull + kMaxAccs, // [kMaxAccs] and read
  kBarriers = kAccEmpty + kMaxAccs
};
static_assert(kBarriers * 8 + 16 <= 512);

constexpr long long kWaitCycles = 4000000000ll;  // ~2 s

struct SkinnyParams {
  __half* out;
  const __half* bias;
  int M, N;
  int n_tiles, k_steps;  // steps of a tile
  int split, per_part;   // parts of a tile (1: whole tiles, CTA b takes b, b + grid, ...), steps of a part (the last: what is left)
};

// q - zp of the 64 k of a column, exact for any byte zp: nibbles become 1024 + q or 64 + q by bit placement, minus 1024 + zp or
// 64 + zp.
__device__ __forceinline__ void integers64(const PackedColumn<kSub>& col, uint32_t shift, uint32_t zp, uint32_t (&out)[32]) {
  const uint32_t lo_off = (0x6400u | zp) * 0x10001u;
  // A conversion: by bit placement (0x5400 | zp << 4) only zero points below 64 fit, and 1024 + zp minus 960 is 5 % slower (8192 x 28672,
  // block 128 41.6 / 43.8 us).
  const uint32_t hi_off = (uint32_t)__half_as_ushort(__uint2half_rn(64u + zp)) * 0x10001u;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint32_t w4[4] = {col.w[c].x, col.w[c].y, col.w[c].z, col.w[c].w};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t x = w4[r] >> shift;
      uint32_t lo, hi;
      asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(lo) : "r"(x), "r"(0x000f000fu), "r"(0x64006400u));
      asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(hi) : "r"(x), "r"(0x00f000f0u), "r"(0x54005400u));
      asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(out[8 * c + r]) : "r"(lo), "r"(lo_off));
      asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(out[8 * c + 4 + r]) : "r"(hi), "r"(hi_off));
    }
  }
}

__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}

template <int BLOCK_SHIFT, bool HAS_ZP>
__global__ void __launch_bounds__(kThreads, 1)
skinny_tc_kernel(const __grid_constant__ CUtensorMap tm_act, const __grid_constant__ CUtensorMap tm_pack,
                 const __grid_constant__ CUtensorMap tm_scale, const __grid_constant__ CUtensorMap tm_zp, const SkinnyParams p) {
  constexpr int kBlocks = BLOCK_SHIFT == 6 ? 2 : 1;  // quantization blocks of a step
  constexpr int kStepAccCols = kBlocks * kRows, kAccs = kAccCols / kStepAccCols;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + kBarOff + kBarriers * 8);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + kBarOff + kBarriers * 8 + 8);
  auto bar = [&](int id) { return base + kBarOff + 8u * (uint32_t)id; };
  auto wait = [&](int id, uint32_t parity, int who) {
    return mbar_wait_bounded(bar(id), parity, abort_flag, &g_skinny_tc_error, who, kWaitCycles);
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // As in the other tensor-core kernels: set-up, the weights' copies and the first dequantized stages run ahead of the preceding
  // kernel's end; activations and the output wait for it.
  asm volatile("griddepcontrol.launch_dependents;");

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bar(kFull + i), 2);       // the packed-tile producer and the meta producer, each with its bytes
      mbar_init(bar(kPackFree + i), 4 + 4);
    }
    for (int i = 0; i < kRing; ++i) {
      mbar_init(bar(kStepFull + i), 4 + 1);
      mbar_init(bar(kMmaDone + i), 1);
    }
    for (int i = 0; i < kMaxAccs; ++i) {
      mbar_init(bar(kAccFull + i), 1);
      mbar_init(bar(kAccEmpty + i), 4);
    }
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // This CTA's work: items b, b + grid, ...; an item is a tile, or the part of one that this CTA of its cluster has.
  const int part = (int)blockIdx.x % p.split, items = p.n_tiles * p.split;
  const int ks0 = part * p.per_part, item_steps = min(p.per_part, p.k_steps - ks0);
  const int my_items = (items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int total_steps = my_items * item_steps;
  float sum[kRows];  // warps 0 to 3, split: this part's sums of column n_l

  if (warp == kActWarp) {
    if (elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");  // activations belong to stream order
      uint32_t s = 0, free_par = 1;  // (the first round finds fresh barriers: the phase before their first one is complete)
      for (int i = 0, ks = ks0; i < total_steps; ++i) {
        if (!wait(kMmaDone + s, free_par, 0x500 | s)) break;
        mbar_arrive_expect_tx(bar(kStepFull + s), kActBytes);
#pragma unroll
        for (int u = 0; u < kSub; ++u)  // past the end of K the copy fills zeros
          tma_load_2d(base + kActOff + s * kActBytes + u * (kRows * 128), &tm_act, ks * kStepK + u * BLOCK_K, 0, bar(kStepFull + s));
        if (++s == kRing) { s = 0; free_par ^= 1u; }
        if (++ks == ks0 + item_steps) ks = ks0;
      }
    }
  } else if (warp == kWeightWarp || warp == kMetaWarp) {
    if (elect_one()) {
      const bool meta = warp == kMetaWarp;
      const uint32_t tx = meta ? (uint32_t)(kBlocks * TILE_N * (HAS_ZP ? 3 : 2)) : (uint32_t)kPackBytes;
      uint32_t s = 0, free_par = 1;
      int tile = (int)blockIdx.x / p.split;
      for (int i = 0, ks = ks0; i < total_steps; ++i) {
        if (!wait(kPackFree + s, free_par, (meta ? 0x520 : 0x510) | s)) break;
        const uint32_t fb = bar(kFull + s);
        mbar_arrive_expect_tx(fb, tx);
        if (!meta) {
          tma_load_2d(base + kPackOff + s * kPackBytes, &tm_pack, ks * kStepK, tile * (TILE_N / 2), fb);
        } else {
          const int row = (ks * kStepK) >> BLOCK_SHIFT;
          tma_load_2d(base + kScaleOff + s * kScaleBytes, &tm_scale, tile * TILE_N, row, fb);
          if (HAS_ZP) tma_load_2d(base + kZpOff + s * kZpBytes, &tm_zp, tile * TILE_N, row, fb);
        }
        if (++s == kStages) { s = 0; free_par ^= 1u; }
        if (++ks == ks0 + item_steps) { ks = ks0; tile += (int)gridDim.x / p.split; }
      }
    }
  } else if (warp == kMmaWarp) {
    // The ring unrolled, the next step polled ahead, as in gemm_tc_kernel.  Blocks are all alike, so this role needs no items.
    if (elect_one() && total_steps > 0) {
      const uint32_t idesc = make_idesc_f16(TILE_N, kRows);
      const uint32_t desc_hi = (uint32_t)(make_sw128_kmajor_desc(0) >> 32);
      const uint32_t act_lo0 = (uint32_t)(make_sw128_kmajor_desc(0) & 0xFFFFFFFFu) | (((base + kActOff) >> 4) & 0x3FFFu);
      const uint32_t a_tmem0 = tmem_base + kDeqCol0;
      uint32_t par = 0, acc = 0, acc_par = 1;
      int left = total_steps;
      bool ready = false;
      for (;; par ^= 1u) {
#pragma unroll
        for (int s = 0; s < kRing; ++s) {
          if (!ready && !wait(kStepFull + s, par, 0x620 | s)) goto mma_done;
          tc_fence_after();
          ready = s + 1 < kRing ? mbar_test_wait(bar(kStepFull + s + 1), par) : mbar_test_wait(bar(kStepFull), par ^ 1u);
          if (!mbar_test_wait(bar(kAccEmpty + acc), acc_par) && !wait(kAccEmpty + acc, acc_par, 0x600 | acc)) goto mma_done;
          tc_fence_after();
#pragma unroll
          for (int u = 0; u < kSub; ++u)
            umma_f16_ts_x4(tmem_base + acc * kStepAccCols + (kBlocks == 2 ? u * kRows : 0), a_tmem0 + (s * kSub + u) * kDeqCols,
                           act_lo0 + ((s * kActBytes + u * (kRows * 128)) >> 4), desc_hi, idesc, kBlocks == 1 && u > 0 ? 1u : 0u);
          umma_commit(bar(kAccFull + acc));
          if (++acc == kAccs) { acc = 0; acc_par ^= 1u; }
          umma_commit(bar(kMmaDone + s));
          if (--left == 0) goto mma_done;
        }
      }
    mma_done:;
    }
  } else if (warp < kFirstDeqWarp) {
    // Scale and add: lane = weight column n of the tile, registers = activation rows.
    const int n_l = warp * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(warp * 32) << 16);
    uint32_t s = 0, full_par = 0, acc = 0, acc_par = 0;
    int tile = (int)blockIdx.x / p.split;
    for (int i = 0; i < my_items; ++i, tile += (int)gridDim.x / p.split) {
      unsigned long long total[kRows / 2];
#pragma unroll
      for (int j = 0; j < kRows / 2; ++j) total[j] = 0ull;  // two fp32 zeros
      for (int k = 0; k < item_steps; ++k) {
        if (!wait(kFull + s, full_par, 0x700 | s)) goto adders_done;
        float scale[kBlocks];
#pragma unroll
        for (int b = 0; b < kBlocks; ++b)
          scale[b] = __half2float(reinterpret_cast<const __half*>(base_ptr + kScaleOff + s * kScaleBytes)[b * TILE_N + n_l]);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kPackFree + s));
        if (++s == kStages) { s = 0; full_par ^= 1u; }
        if (!wait(kAccFull + acc, acc_par, 0x720 | acc)) goto adders_done;
        tc_fence_after();
        uint32_t r[kBlocks][kRows];
        if constexpr (kBlocks == 2) tmem_ld_32x32b_x32(lane_base + acc * kStepAccCols, reinterpret_cast<uint32_t (&)[32]>(r));
        else tmem_ld_32x32b_x16(lane_base + acc * kStepAccCols, r[0]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kAccEmpty + acc));
        if (++acc == kAccs) { acc = 0; acc_par ^= 1u; }
#pragma unroll
        for (int b = 0; b < kBlocks; ++b) {
          const unsigned long long s2 = pack2(scale[b], scale[b]);
#pragma unroll
          for (int j = 0; j < kRows / 2; ++j)
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(total[j]) : "l"(pack2(__uint_as_float(r[b][2 * j]), __uint_as_float(r[b][2 * j + 1]))), "l"(s2));
        }
      }
#pragma unroll
      for (int j = 0; j < kRows / 2; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(sum[2 * j]), "=f"(sum[2 * j + 1]) : "l"(total[j]));
      if (p.split > 1) break;  // the cluster adds its parts up after the role branches
      if (i == 0) asm volatile("griddepcontrol.wait;" ::: "memory");  // the output belongs to stream order
      // lanes pair up (n even / odd): the even one stores the even rows of both columns, the odd one the odd rows
      const int n = tile * TILE_N + n_l, odd = lane & 1;
      const uint32_t pick = trade_selector(odd);
      const bool n_ok = (n | 1) < p.N;  // N is a multiple of 16: the pair is in or out together
      // the bias is added to the rounded result in fp16, as a separate `output += bias` does
      const bool add_bias = p.bias != nullptr && n_ok;
      const __half2 bias2 = add_bias ? *reinterpret_cast<const __half2*>(p.bias + (n & ~1)) : __half2();
#pragma unroll
      for (int j = 0; j < kRows; j += 2) {
        const uint32_t traded = trade_rows(__float_as_uint(sum[j]), __float_as_uint(sum[j + 1]), pick);
        __half2 v = *reinterpret_cast<const __half2*>(&traded);
        if (add_bias) v = __hadd2(v, bias2);
        const int m = j + odd;
        if (n_ok && m < p.M) *reinterpret_cast<__half2*>(p.out + (size_t)m * p.N + (n & ~1)) = v;
      }
    }
  adders_done:;
  } else {
    // Dequantizers: as in gemm_tc_kernel, thread = weight column n of the tile.
    const int group = (warp - kFirstDeqWarp) / 4;
    const int n_l = 32 * (warp & 3) + lane;
    const int np_l = 8 * (n_l >> 4) + (n_l & 7);
    const uint32_t shift = (n_l & 8) ? 8u : 0u;
    const uint32_t tmem_row = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + kDeqCol0;
    for (int it = group; it < total_steps; it += kGroups) {
      const int s = it % kStages, d = it % kRing;
      if (!wait(kMmaDone + d, ((it / kRing) & 1) ^ 1u, 0x810 | d)) break;
      if (!wait(kFull + s, (it / kStages) & 1, 0x800 | s)) break;
      tc_fence_after();
      const uint8_t* pk = base_ptr + kPackOff + s * kPackBytes + np_l * kStepK;
      const uint8_t* zp_tile = base_ptr + kZpOff + s * kZpBytes;
      PackedColumn<kSub> sub[kSub];
#pragma unroll
      for (int u = 0; u < kSub; ++u) sub[u].load(pk, u, n_l);
#pragma unroll
      for (int u = 0; u < kSub; ++u) {
        uint32_t out[32];
        integers64(sub[u], shift, HAS_ZP ? (uint32_t)zp_tile[(kBlocks == 2 ? u : 0) * TILE_N + n_l] : 8u, out);
        tmem_st_32x32b_x32(tmem_row + (uint32_t)((d * kSub + u) * kDeqCols), out);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar(kStepFull + d));
        mbar_arrive(bar(kPackFree + s));
      }
    }
  }

  if (p.split > 1) {
    // Split K: part q of the cluster owns `slice4` groups of four rows; every part stores the others' rows of its sums into their
    // shared memory, over the activation ring, [part][row group][column] with four rows of a column as 16 bytes, and adds up
    // its own rows in part order (see gemm_tc_kernel).
    asm volatile("griddepcontrol.wait;" ::: "memory");  // all warps store to the output
    __syncwarp();
    cluster_sync_all();  // every part has read its last accumulator, so the activation rings are idle
    const int slice4 = (kRows / 4 + p.split - 1) / p.split;
    if (warp < kFirstDeqWarp) {
      const int n_l = warp * 32 + lane;
#pragma unroll
      for (int g = 0; g < kRows / 4; ++g) {
        const int owner = g / slice4;
        st_shared_cluster_v4(map_to_cta(base + kActOff + (uint32_t)(((part * slice4 + g - owner * slice4) * TILE_N + n_l) * 16), (uint32_t)owner),
                             __float_as_uint(sum[4 * g]), __float_as_uint(sum[4 * g + 1]), __float_as_uint(sum[4 * g + 2]),
                             __float_as_uint(sum[4 * g + 3]));
      }
    }
    cluster_sync_all();
    const int g0 = part * slice4, mine = min(slice4, (p.M + 3) / 4 - g0);
    const float4* src = reinterpret_cast<const float4*>(base_ptr + kActOff);
    for (int idx = threadIdx.x; idx < mine * TILE_N; idx += kThreads) {  // whole warps
      const int n = (int)blockIdx.x / p.split * TILE_N + (idx % TILE_N);
      float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
      for (int q = 0; q < p.split; ++q) {
        const float4 f = src[q * slice4 * TILE_N + idx];
        t.x += f.x;
        t.y += f.y;
        t.z += f.z;
        t.w += f.w;
      }
      // lanes pair up (n even / odd): the even one stores rows 0 and 1 of both columns, the odd one rows 2 and 3
      const int odd = lane & 1;
      const float got0 = __shfl_xor_sync(0xffffffffu, odd ? t.x : t.z, 1);
      const float got1 = __shfl_xor_sync(0xffffffffu, odd ? t.y : t.w, 1);
      __half2 h0 = odd ? __floats2half2_rn(got0, t.z) : __floats2half2_rn(t.x, got0);
      __half2 h1 = odd ? __floats2half2_rn(got1, t.w) : __floats2half2_rn(t.y, got1);
      const int m = 4 * (g0 + idx / TILE_N) + 2 * odd;
      if (n < p.N) {
        if (p.bias) {
          const __half2 b = *reinterpret_cast<const __half2*>(p.bias + (n & ~1));
          h0 = __hadd2(h0, b);
          h1 = __hadd2(h1, b);
        }
        __half* dst = p.out + (size_t)m * p.N + (n & ~1);
        if (m < p.M) *reinterpret_cast<__half2*>(dst) = h0;
        if (m + 1 < p.M) *reinterpret_cast<__half2*>(dst + p.N) = h1;
      }
    }
  }

  // ---- teardown ----
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) __nanosleep(50000);  // let copies in flight land
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

using Kern = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, SkinnyParams);

// Clusters of `split` CTAs that are resident at once on the current device (0: it cannot say).
int resident_clusters(Kern kern, int split) {
  static std::atomic<int> cache[kMaxSplit + 1][64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const bool cached = dev >= 0 && dev < 64;
  int n = cached ? cache[split][dev].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sm_count() / split * split);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 0) {
    cudaGetLastError();
    return 0;
  }
  if (cached && n > 0) cache[split][dev].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace

bool skinny_tc_takes(int block, bool colwise, int M, int N, int K, const void* scales, const void* zp) {
  return colwise && block >= 64 && M >= 1 && M <= 16 && K % 64 == 0 && N % 16 == 0 && reinterpret_cast<uintptr_t>(scales) % 16 == 0 &&
         reinterpret_cast<uintptr_t>(zp) % 16 == 0;
}

// Up to eight rows the decode kernel's CTAs take 16 columns at a time, whose end costs a barrier and the addition of eight partial
// sums, and one or two of its eight warps may have a group of steps more than the others; this kernel takes 128 columns, and time
// that hardly depends on the rows, but a launch that cannot start early costs 2.9 us in place of 1.4.  The kernel must not depend on whether
// it can (the results would), so that the lines lie where the two are equal in the geometric mean of both kinds of launches.
// K in whole groups from 2048 on stays with the decode kernel: layers of such K may share a launch there, with the bits of their own
// calls.  Measured on B200, decode kernel / this one with the early weight fetch (without), us, block 64 with zero points, K x N:
//   K < 512: M = 1 128 x 11008 0.82 of the time, 64 x 28672 3.4 / 3.1 (4.3 / 4.4), 256 x 18944 1.00 (there), 64 x 4096 1.8 / 2.1
//     (2.6 / 3.6: there); M = 3 64 x 2048 2.1 / 2.0 (2.9 / 3.5: there), 192 x 6144 3.3 / 2.3 (4.2 / 4.0); M = 5 192 x 2048 2.6 / 2.2 (3.4 / 3.9);
//     M = 8 256 x 2048 2.9 / 2.3 (3.7 / 3.9), 448 x 2048 3.0 / 2.7 (3.9 / 4.5); two rounds of tiles: M = 8 192 x 28672 6.3 / 4.1 (7.4 / 5.8),
//     M = 3 320 x 22528 0.95.  (The generic kernel, which rounds the weights to fp16, takes 3.2 for 64 x 28672 and 4.3 for 192 x 28672
//     with either launch: slower than this one with the early fetch, faster without.)
//   512 to 703: M = 5 512 x 6144 3.8 / 2.7 (4.6 / 4.6), 512 x 11008 4.6 / 3.5 (6.1 / 5.5); M = 8 512 x 2048 3.0 / 2.6 (3.8 / 4.5: there);
//     two rounds of tiles: M = 5 512 x 22528 0.94 of the time, M = 8 640 x 28672 0.85, 768 x 28672 0.90
//   704 to 2047: M = 8 768 x 8192 4.3 / 3.2 (5.7 / 6.1), 1024 x 6144 4.6 / 3.8 (6.0 / 6.8), 1536 x 6144 5.1 / 5.1 (6.7 / 7.1: there);
//     M = 5 768 x 11008 5.1 / 4.0 (6.6 / 6.2); M = 6 1536 x 14336 7.5 / 6.6 (9.3 / 8.4), 1536 x 18944 7.5 / 7.3 (9.3 / 8.7), 1792 x 11008 1.1
//   2048 to 4095: M = 7 2112 x 3072 5.6 / 5.2 (7.3 / 6.7), M = 8 3200 x 1024 0.90, 3200 x 11008 1.05 (86 tiles: 62 SMs without work); M = 6 1.0 to 1.1
//   from 4096 on, few columns: M = 5 5184 x 2048 6.7 / 5.9 (7.6 / 7.7), M = 8 5184 x 4096 9.3 / 7.8 (11.0 / 9.3), 6208 x 1024 8.5 / 5.4 (10.1 / 7.6);
//     M = 3 6208 x 1024 6.3 / 5.4 (7.5 / 7.6), 8256 x 1024 7.9 / 6.2, 8256 x 2048 9.0 / 7.3; M = 6 8256 x 4096 12.1 / 9.9; many columns:
//     M = 8 8256 x 8192 18.4 / 15.1, 8256 x 18944 0.85 of the time; M = 6 8256 x 6144 14.3 / 14.3
bool skinny_tc_is_faster(int M, int N, int K) {
  if (K >= 2048 && K % 256 == 0) return false;
  const int sms = sm_count(), tiles = (N + TILE_N - 1) / TILE_N;
  const bool few = N <= 32 * sms;
  if (M < 3) return K < 256 && N > 64 * sms;
  if (K < 512) return M >= (few ? (K < 256 ? 5 : 7) : tiles <= sms || K <= 256 ? 3 : 5);
  if (K < 704) return !few && M >= (tiles <= sms ? 3 : 5);
  if (tiles > sms) return false;
  if (K < 1152) return N > 64 * sms ? M >= 5 : !few && M >= 7;
  if (tiles * 2 > sms && tiles * 10 < sms * 7) return false;  // neither split nor enough tiles for the SMs
  if (K < 2048) return N > 64 * sms && M >= 6;
  if (K < 4096 || !few) return M >= 7;
  return M >= (N > 16 * sms ? 6 : K < 6144 ? 5 : 3);
}

std::string launch_skinny_tc(int block, int M, int N, int K, cudaStream_t stream, const __half* a, const uint8_t* packed,
                             const __half* scales, const uint8_t* zp, __half* out, const __half* bias, unsigned flags) {
  SkinnyParams p{};
  p.out = out; p.bias = bias; p.M = M; p.N = N;
  p.n_tiles = (N + TILE_N - 1) / TILE_N;
  p.k_steps = (K + kStepK - 1) / kStepK;
  const uint32_t meta_rows = block == 64 ? 2 : 1;
  CUtensorMap tm_act, tm_pack, tm_scale, tm_zp;
  bool ok = encode_tensor_map_2d(&tm_act, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a, (uint64_t)K, (uint64_t)M, BLOCK_K, kRows,
                                 CU_TENSOR_MAP_SWIZZLE_128B);
  ok = ok && encode_tensor_map_2d(&tm_pack, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, packed, (uint64_t)K, (uint64_t)(N / 2), kStepK, TILE_N / 2,
                                  CU_TENSOR_MAP_SWIZZLE_128B);
  ok = ok && encode_tensor_map_2d(&tm_scale, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, scales, (uint64_t)N, (uint64_t)(K / block), TILE_N,
                                  meta_rows, CU_TENSOR_MAP_SWIZZLE_NONE);
  ok = ok && encode_tensor_map_2d(&tm_zp, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, zp ? zp : packed, (uint64_t)N, (uint64_t)(K / block), TILE_N,
                                  meta_rows, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (!ok) return "cuTensorMapEncodeTiled failed";
  Kern kern = block == 64 ? (zp ? (Kern)skinny_tc_kernel<6, true> : (Kern)skinny_tc_kernel<6, false>)
                          : (zp ? (Kern)skinny_tc_kernel<7, true> : (Kern)skinny_tc_kernel<7, false>);
  static std::atomic<int> granted[4][64];
  cudaError_t e = ensure_dynamic_smem(kern, kSmemBytes, granted[(block == 64 ? 0 : 2) + (zp ? 1 : 0)]);
  if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
  // As many parts of at least 512 k as there are SMs for; in two only from 2048 k on (see short_k_parts of blkq4_gemm_tc.cu).
  const int sms = sm_count();
  p.split = 1;
  p.per_part = p.k_steps;
  for (int parts = 2; parts <= kMaxSplit && p.n_tiles * 2 <= sms; ++parts) {
    const int per = (p.k_steps + parts - 1) / parts, split = (p.k_steps + per - 1) / per;
    if (split < 2 || per * kStepK < 512 || p.n_tiles * split > sms) continue;
    p.split = split;
    p.per_part = per;
  }
  if (p.split == 2 && K < 2048) { p.split = 1; p.per_part = p.k_steps; }
  while (p.split > 1 && resident_clusters(kern, p.split) < p.n_tiles) {  // a group of SMs holds whole clusters only
    p.per_part = (p.k_steps + p.split - 2) / (p.split - 1);
    p.split = (p.k_steps + p.per_part - 1) / p.per_part;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = p.split > 1 ? attr : attr + 1;
  cfg.numAttrs = (p.split > 1 ? 1 : 0) + ((flags & BLKQ4_GEMM_EARLY_WEIGHT_FETCH) ? 1 : 0);
  cfg.gridDim = dim3(p.split > 1 ? p.n_tiles * p.split : p.n_tiles < sms ? p.n_tiles : sms);
  e = cudaLaunchKernelEx(&cfg, kern, tm_act, tm_pack, tm_scale, tm_zp, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return std::string(cudaGetErrorString(e));
  return std::string();
}

int clear_skinny_tc_error(cudaStream_t stream) {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_skinny_tc_error) != cudaSuccess) return -1;
  return cudaMemsetAsync(p, 0, sizeof(int), stream) == cudaSuccess ? 0 : -1;
}

int read_skinny_tc_error() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_skinny_tc_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // namespace blkq4
