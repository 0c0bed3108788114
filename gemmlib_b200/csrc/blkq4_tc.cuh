// Pieces shared by the tensor-core W4A16 kernels (one CTA per tile, and CTA pairs): tile constants,
// tcgen05 / tensor-memory PTX wrappers, operand descriptors and the dequantization of one 64-k step of
// one weight column.
#pragma once

#include <cstdint>

#include "blkq4_common.cuh"
#include "blkq4_tma.cuh"

namespace blkq4 {
namespace tc {

constexpr int TILE_N = 128;       // weight columns per CTA tile (UMMA M of one CTA)
constexpr int BLOCK_K = 64;       // k per pipeline step: one 128-byte swizzle row of fp16
constexpr int kDeqCols = BLOCK_K / 2;  // TMEM columns of one dequantized stage: 2 fp16 per column
constexpr int kPackTileBytes = (TILE_N / 2) * BLOCK_K;  // 4 KB: 64 packed columns x 64 bytes
constexpr int kScaleTileBytes = 1024;
constexpr int kZpTileBytes = 512;

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// First operand from tensor memory: 128 lanes (rows) x 8 columns per 16 k, two fp16 per column.
// The four MMAs of one 64-k step: operand A advances 8 TMEM columns, operand B two
// descriptor units (32 bytes) per 16 k.  Only the first may overwrite the accumulator.
__device__ __forceinline__ void umma_f16_ts_x4(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 b0, b1, b2, b3;\n\t.reg .b32 l1, l2, l3, a1, a2, a3;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 q, 0, 0;\n\t"
      "add.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "mov.b64 b0, {%2, %3};\n\tmov.b64 b1, {l1, %3};\n\tmov.b64 b2, {l2, %3};\n\tmov.b64 b3, {l3, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b0, %4, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %4, q;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %4, q;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %4, q;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Two accumulator values of one weight column n, activation rows m and m + 1, rounded to fp16 and traded with the lane of
// the other column of the pair (lanes n even / odd): the even lane gets row m of both columns, the odd one row m + 1.
// `pick` is trade_selector(n odd).  One conversion, shuffle and byte permutation for two values.
__device__ __forceinline__ uint32_t trade_selector(int odd) { return odd ? 0x3276u : 0x5410u; }
__device__ __forceinline__ uint32_t trade_rows(uint32_t row0, uint32_t row1, uint32_t pick) {
  const __half2 own = __floats2half2_rn(__uint_as_float(row0), __uint_as_float(row1));
  const uint32_t mine = *reinterpret_cast<const uint32_t*>(&own);
  return __byte_perm(mine, __shfl_xor_sync(0xffffffffu, mine, 1), pick);
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `local_addr` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_shared_cluster_v4(uint32_t cluster_addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(cluster_addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes
// (64 fp16) with the 128-byte swizzle, rows contiguous, tile base 1024-byte aligned:
// start address >> 4 in bits 0-13, leading byte offset (unused for swizzled K-major) = 1
// in bits 16-29, stride byte offset 1024 >> 4 (one 8-row group) in bits 32-45, descriptor
// version 1 in bits 46-47, layout type 2 (SWIZZLE_128B) in bits 61-63.
__device__ __forceinline__ uint64_t make_sw128_kmajor_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) |
         (2ull << 61);
}
// Instruction descriptor, kind::f16: fp32 accumulator (bits 4-5 = 1), fp16 A and B
// (formats 0), both K-major, N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ inline uint32_t make_idesc_f16(int umma_m, int umma_n) {
  return (1u << 4) | ((uint32_t)(umma_n >> 3) << 17) | ((uint32_t)(umma_m >> 4) << 24);
}


// One 64-k sub-step of weight column n_l of a tile (a step holds KSUB of them): `load` reads the column's 64
// packed bytes and its scales / zero points from the stage in shared memory, `emit` produces the 32 fp16
// pairs of the dequantized stage, out[j] = k pair (2j, 2j + 1).  Numerics are the reference kernel's: fp16(16 + q)
// by bit placement, then fma.rn.f16 with rn(scale * (-16 - zp)).
// Block size and zero points are template parameters and loading is separate from converting so that all
// loads of a step are issued back to back: with a runtime block size every 16-k chunk had its own
// dependent scale load and a branch on the zero points, and a step cost a dequantizer group ~2300 cycles of
// mostly latency (M = 17, K = 8192, N = 28672, block 128: 46.1 us against 26.3 us without the conversion).
template <int KSUB>
struct PackedColumn {
  uint4 w[4];
  // `pk` points at the packed column; 128-byte rows are stored with the 128-byte swizzle (chunk c of packed
  // column r lies at c ^ (r % 8)), so that the eight columns a quarter-warp reads fall on different banks
  __device__ __forceinline__ void load(const uint8_t* pk, int sub, int n_l) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int cc = sub * 4 + c;
      w[c] = *reinterpret_cast<const uint4*>(pk + (KSUB == 2 ? ((cc ^ (n_l & 7)) * 16) : cc * 16));
    }
  }
  // Column n0's nibbles sit at bits 0-3 / 16-19 (k = 2r, 2r+1) and 4-7 / 20-23 (k = 2r+8, 2r+9) of word r, column
  // n0 + 8's eight bits further up; fp16(16 + q) by bit placement needs them at bits 6-9 / 22-25.  One
  // rotation per operand does it (instead of a shift to this thread's nibbles and a second one into
  // place): left by 6 / 2 for n0, by 30 / 26 (= right by 2 / 6) for n0 + 8; what wraps around falls
  // outside the mask.
  __device__ __forceinline__ static uint32_t half16plus(uint32_t w, uint32_t rot) {
    return (__funnelshift_l(w, w, rot) & 0x03c003c0u) | 0x4c004c00u;
  }
};

template <bool COLWISE, int BLOCK_SHIFT, bool HAS_ZP, int KSUB>
struct DequantSub;

// Column-wise blocks: meta tile = rows of 128 columns, one row per block of k.
template <int BLOCK_SHIFT, bool HAS_ZP, int KSUB>
struct DequantSub<true, BLOCK_SHIFT, HAS_ZP, KSUB> : PackedColumn<KSUB> {
  static constexpr int kBlocks = BLOCK_SHIFT >= 6 ? 1 : (BLOCK_K >> BLOCK_SHIFT);  // of a sub-step
  uint32_t s[kBlocks], z[kBlocks];
  __device__ __forceinline__ void load(const uint8_t* pk, int sub, const uint8_t* sc_tile, const uint8_t* zp_tile, int n_l) {
    PackedColumn<KSUB>::load(pk, sub, n_l);
    const int row0 = BLOCK_SHIFT > 6 ? 0 : sub * kBlocks;
#pragma unroll
    for (int b = 0; b < kBlocks; ++b) {
      s[b] = reinterpret_cast<const unsigned short*>(sc_tile)[(row0 + b) * TILE_N + n_l];
      z[b] = HAS_ZP ? (uint32_t)zp_tile[(row0 + b) * TILE_N + n_l] : 8u;
    }
  }
  __device__ __forceinline__ void emit(const uint8_t*, const uint8_t*, int, int, uint32_t rot_lo, uint32_t rot_hi,
                                       uint32_t (&out)[32]) const {
#pragma unroll
    for (int c = 0; c < 4; ++c) {  // 16-byte chunk: k in [16 c, 16 c + 16) of the sub-step
      const int b = BLOCK_SHIFT >= 6 ? 0 : ((c * 16) >> BLOCK_SHIFT);
      const uint32_t sc2 = s[b] | (s[b] << 16);
      // fp16(-16 - z) by bit placement (0xcc00 is -16.0, mantissa step 1/64), times the scale
      const uint32_t nz = 0xcc00u | (z[b] << 6);
      const uint32_t of2 = hmul2_u32(sc2, nz | (nz << 16));
      const uint32_t w4[4] = {this->w[c].x, this->w[c].y, this->w[c].z, this->w[c].w};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        // chunk c, word r: k = 16 c + 2 r (+1) -> column 8 c + r; k + 8 -> column 8 c + 4 + r
        out[8 * c + r] = hfma2_u32(sc2, this->half16plus(w4[r], rot_lo), of2);
        out[8 * c + 4 + r] = hfma2_u32(sc2, this->half16plus(w4[r], rot_hi), of2);
      }
    }
  }
};

// Row-wise blocks: meta tile = (128 / block) rows of the step's k, permuted per 16 as 0 1 8 9 2 3 10 11 ...
// (scales) and 0 8 1 9 2 10 3 11 ... (zero points).
template <int BLOCK_SHIFT, bool HAS_ZP, int KSUB>
struct DequantSub<false, BLOCK_SHIFT, HAS_ZP, KSUB> : PackedColumn<KSUB> {
  __device__ __forceinline__ void load(const uint8_t* pk, int sub, const uint8_t*, const uint8_t*, int n_l) {
    PackedColumn<KSUB>::load(pk, sub, n_l);
  }
  __device__ __forceinline__ void emit(const uint8_t* sc_tile, const uint8_t* zp_tile, int sub, int n_l, uint32_t rot_lo,
                                       uint32_t rot_hi, uint32_t (&out)[32]) const {
    const int mr = n_l >> BLOCK_SHIFT;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int cc = sub * 4 + c;
      const uint4* sp = reinterpret_cast<const uint4*>(sc_tile + mr * (128 * KSUB) + cc * 32);
      const uint4 s0 = sp[0], s1 = sp[1];
      const uint32_t sw[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
      uint4 zv = make_uint4(0x08080808u, 0x08080808u, 0x08080808u, 0x08080808u);
      if (HAS_ZP) zv = *reinterpret_cast<const uint4*>(zp_tile + mr * (64 * KSUB) + cc * 16);
      const uint32_t zw[4] = {zv.x, zv.y, zv.z, zv.w};
      const uint32_t w4[4] = {this->w[c].x, this->w[c].y, this->w[c].z, this->w[c].w};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t nz_lo = ((zw[r] << 6) & 0x03c003c0u) | 0xcc00cc00u;  // fp16(-16 - z)
        const uint32_t nz_hi = ((zw[r] >> 2) & 0x03c003c0u) | 0xcc00cc00u;
        out[8 * c + r] = hfma2_u32(sw[2 * r], this->half16plus(w4[r], rot_lo), hmul2_u32(sw[2 * r], nz_lo));
        out[8 * c + 4 + r] = hfma2_u32(sw[2 * r + 1], this->half16plus(w4[r], rot_hi), hmul2_u32(sw[2 * r + 1], nz_hi));
      }
    }
  }
};

// Calls fn(block shift, zero points) with both as compile-time constants.
template <int V>
struct IntC {
  static constexpr int value = V;
};
template <typename Fn>
__device__ __forceinline__ void with_block_shift(int block_shift, int has_zp, Fn&& fn) {
  if (has_zp) {
    if (block_shift == 7) fn(IntC<7>{}, IntC<1>{});
    else if (block_shift == 6) fn(IntC<6>{}, IntC<1>{});
    else if (block_shift == 5) fn(IntC<5>{}, IntC<1>{});
    else fn(IntC<4>{}, IntC<1>{});
  } else {
    if (block_shift == 7) fn(IntC<7>{}, IntC<0>{});
    else if (block_shift == 6) fn(IntC<6>{}, IntC<0>{});
    else if (block_shift == 5) fn(IntC<5>{}, IntC<0>{});
    else fn(IntC<4>{}, IntC<0>{});
  }
}

}  // namespace tc
}  // namespace blkq4
