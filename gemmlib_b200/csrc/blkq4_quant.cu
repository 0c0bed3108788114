// Fused blockwise 4-bit quantization + prepack for sm_100a.
//
// One kernel per call replaces the reference's three (block_quantize_kernel,
// prepack_weights_kernel, prepack_scales_kernel; reference
// src/mickey/blk_q4/f16_quant_sm80.cuh:593-653) and its three temporary device
// buffers (src/blkq4_f16_gemm_sm80.cu:282-290).  It is memory bound: every fp16
// weight is read from HBM once and the packed bytes, scales and zero points are
// written once in their final order.  Output bytes are bit-identical to the
// reference's.
//
// A thread owns one 16-byte packed chunk: 16 consecutive k of the columns n0 and n0 + 8, i.e. 32 contiguous
// bytes of each of two weight rows, which it keeps in registers from the load to the store.  A warp owns 64 k of
// 16 columns (128 k of 8 columns for column-wise blocks of 128), so that a load instruction covers whole
// 128-byte lines and the meta entries of a warp share sectors.
//
// What the arithmetic may cost: at HBM's rate an SM moves 22 bytes a cycle (6.5 TB/s, 148 SMs, 1.97 GHz), i.e. finishes
// 9 weights of 2.5 bytes, so with every issue slot used (128 threads a cycle) the budget is 14 instructions per
// weight.  The column-wise kernel executes 9.7 (13.7 M warp instructions for 45 M weights), ~5 of them in quantize_pair
// and assemble_word, and issues in 65 % of the cycles.  Measured on B200 (4096 x 11008, block 64, zero points, 114 MB):
// 28.5 us with 14 in the conversion alone - float-to-integer conversions and min / max on quarter- and half-rate pipes,
// the scale's divisions repeated by every lane of a block - and 21.5 us now (0.81 of the measured copy bandwidth).
//
// A CTA is short: it loads, waits, computes and leaves, so small ones keep the SM's slots turning over more evenly.  CTAs of
// 128 threads, ten of them on an SM (48 registers), against 256, us: column-wise 4096 x 11008 22.0 / 21.5, 8192 x 28672
// block 128 101.7 / 94.8; row-wise 11008 x 4096 block 32 28.1 / 25.0, 4096 x 11008 block 64 29.0 / 24.8.  Twelve on an SM
// (40 registers, spills) 21.5, 101.9, 26.7, 25.8.  Of the kernels with 48 registers only column-wise block 16 spills, 4 bytes
// (8 with unaligned rows); 256 threads and 42 registers against that: 4096 x 11008 22.7 / 22.2, symmetric 20.9 / 20.4, 8192 x 28672
// 106.8 / 105.7.
#include "blkq4_common.cuh"

namespace blkq4 {
namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr unsigned kMaxGridY = 32768;

// Both kernels are launched with programmatic stream serialization: their CTAs become resident, and the launch's own
// latency passes, while the preceding kernel ends (or, where that kernel lets its successor start early, while it still
// runs); nothing is read or written before it has completed.  Measured on B200, seven weights of a decoder block (4096, 11008;
// block 64, zero points) 117.1 us without it, 104.9 with; row-wise 11008 x 4096, block 32 29.0 / 26.7.
// They execute no griddepcontrol.launch_dependents: a GEMM with BLKQ4_GEMM_EARLY_WEIGHT_FETCH right behind a quantizer would
// then read packed weights that are not written yet.  It would gain nothing either (quantizer behind quantizer, with / without:
// 106.1 / 104.9 us a block, row-wise 26.7 / 26.7; 4096 x 4096, block 16 10.8 / 10.8).
__device__ __forceinline__ void start_in_stream_order() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Scale and zero point from a block's range.  Same float operation sequence as
// the reference's range2scalezp (f16_quant_sm80.cuh:96-122): IEEE division,
// roundf (halves away from zero), clamp to [0, 15], fp32 -> fp16 round-to-nearest.
__device__ __forceinline__ void range_to_scale_zp(float mn, float mx, __half& scale, uint8_t& zp) {
  mn = fminf(mn, 0.0f);
  mx = fmaxf(mx, 0.0f);
  const float scale_f = __fdiv_rn(mx - mn, 15.0f);
  float zpf = mn;
  if (scale_f != 0.0f) zpf = 0.0f - __fdiv_rn(mn, scale_f);
  if (zpf < 0.0f) {
    zp = 0;
  } else if (zpf > 15.0f) {
    zp = 15;
  } else {
    zp = (uint8_t)roundf(zpf);
  }
  scale = __float2half_rn(scale_f);
}

// Symmetric case, reference range2scale (f16_quant_sm80.cuh:124-135): the
// extreme of larger magnitude, sign kept, over -8.  The reference scans a block
// sequentially with "v < min", so for an all-zero block its min is the first
// element it meets, sign of zero included; `first` reproduces that.
__device__ __forceinline__ __half range_to_scale(float mn, float mx, float first) {
  float m = fabsf(mx) > fabsf(mn) ? mx : mn;
  if (mn == 0.0f && mx == 0.0f) m = first;
  return __float2half_rn(m * -0.125f);
}

// Scale, zero point (8 when symmetric) and the fp32 reciprocal of the rounded scale.
__device__ __forceinline__ void block_params(float mn, float mx, float first, bool has_zp, __half& scale, uint8_t& zp,
                                             float& recip) {
  zp = 8;
  if (has_zp) range_to_scale_zp(mn, mx, scale, zp);
  else scale = range_to_scale(mn, mx, first);
  const float s = __half2float(scale);
  recip = (s != 0.0f) ? __fdiv_rn(1.0f, s) : 0.0f;
}

__device__ __forceinline__ unsigned long long pack_f32x2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}

// Two weights v at once: 15 - q with q = clamp(round_half_away(v * r + zp), 0, 15), each in a 16-bit field with
// 15 - q at bits POS .. POS + 3, fraction bits below and zeros above.  nr2 and nz2 are -r and -zp.
//
// The reference's expression (f16_quant_sm80.cuh:295-296) is compiled by nvcc with its default fused multiply-add
// contraction; the fma is explicit here and gives -x for x = v * r + zp.  For x >= 0 rounding halves away from zero
// is floor(x + 0.5), and negative x end at 0 either way.  With n = floor((x + 0.5) * 2^POS), adding
// 1.5 * 2^(23 - POS) + 15.5 - 2^-POS with rounding toward +infinity leaves 16 * 2^POS - 1 - n in the low mantissa
// bits (the sum is positive and its last place is 2^-POS), so one packed fp32 addition does the rounding and the
// conversion; the low 16 bits are that integer in two's complement (|x| < 38: a subnormal scale may be off by
// half of itself), which a packed 16-bit minimum with the negative values flushed to zero clamps to
// [0, 16 * 2^POS - 1].  Why 15 - q: a NaN (a NaN weight, or an infinite one, whose block has r = 0) has all low
// bits set, which is flushed to zero, and the reference's min(15, NaN) makes it q = 15.
template <int POS>
__device__ __forceinline__ uint32_t quantize_pair(uint32_t v, unsigned long long nr2, unsigned long long nz2) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
  constexpr float kMagic = (float)(1.5 * (1 << (23 - POS)) + 15.5 - 1.0 / (1 << POS));
  unsigned long long x;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(x) : "l"(pack_f32x2(f.x, f.y)), "l"(nr2), "l"(nz2));
  asm("add.rp.f32x2 %0, %1, %2;" : "=l"(x) : "l"(x), "l"(pack_f32x2(kMagic, kMagic)));
  uint32_t lo, hi, q;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(x));
  constexpr uint32_t kMax = (16u << POS) - 1u;
  asm("min.relu.s16x2 %0, %1, %2;" : "=r"(q) : "r"(__byte_perm(lo, hi, 0x5410)), "r"(kMax | (kMax << 16)));
  return q;
}

// (a & mask) | (b & ~mask)
__device__ __forceinline__ uint32_t select_bits(uint32_t a, uint32_t b, uint32_t mask) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xe4;" : "=r"(d) : "r"(a), "r"(b), "r"(mask));
  return d;
}

// One packed word (reference dev_prepack_weights, f16_quant_sm80.cuh:362-417) of k = 2r, 2r + 1, 2r + 8, 2r + 9:
// nibbles, from bit 0, of (2r, n0) (2r + 8, n0) (2r, n0 + 8) (2r + 8, n0 + 8), the same for 2r + 1 from bit 16.
// a0, b0: quantize_pair<4> of k pair 2r, columns n0 and n0 + 8; a1, b1: quantize_pair<8> of k pair 2r + 8.  All
// 32 bits come out complemented (~0xe4 = 0x1b), which turns every 15 - q into q.
__device__ __forceinline__ uint32_t assemble_word(uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1) {
  const uint32_t a = select_bits(a0, a1, 0x00ff00ffu), b = select_bits(b0, b1, 0x00ff00ffu);
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0x1b;" : "=r"(d) : "r"(a >> 4), "r"(b << 4), "r"(0x00ff00ffu));
  return d;
}

// 16 halves of a weight row.  ALIGNED: 16-byte loads.  Otherwise the row starts at any even address: seven aligned
// words and the two halves of the eighth that are left over, shifted into place by one byte permutation each; nothing
// outside the 32 bytes is read, and lanes of both alignments (an odd leading dimension) run the same instructions.
// Measured on B200, 8192 x 28672, block 64, base at an odd half: sixteen 2-byte loads 251 us, staged in shared
// memory 194, this 156 (16-byte loads of aligned rows: 100).
template <bool ALIGNED>
__device__ __forceinline__ void load_row16(const __half* src, uint32_t (&v)[8]) {
  if (ALIGNED) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(src)), y = __ldg(reinterpret_cast<const uint4*>(src) + 1);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
  } else {
    const unsigned short* s = reinterpret_cast<const unsigned short*>(src);
    const bool odd = reinterpret_cast<uintptr_t>(src) & 2;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(s + (odd ? 1 : 0));
    uint32_t w[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) w[i] = __ldg(q + i);
    const uint32_t x = __ldg(s + (odd ? 0 : 14)), y = __ldg(s + 15);  // odd: the first and the last half; else the last two
    const uint32_t sel = odd ? 0x5432u : 0x7654u;
    v[0] = __byte_perm(x << 16, w[0], sel);
#pragma unroll
    for (int i = 1; i < 7; ++i) v[i] = __byte_perm(w[i - 1], w[i], sel);
    v[7] = __byte_perm(w[6], odd ? y : (x | (y << 16)), sel);
  }
}

// fp16 minimum / maximum of two pairs (exact; NaNs are skipped as in the reference's "v < min" scan).
__device__ __forceinline__ uint32_t hmin2_u32(uint32_t a, uint32_t b) {
  const __half2 r = __hmin2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t hmax2_u32(uint32_t a, uint32_t b) {
  const __half2 r = __hmax2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ float half_bits_to_float(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }

// ---- column-wise blocks -------------------------------------------------------------------------------
// The BLOCK / 16 lanes of a quantization block are neighbours along k; its range is a shuffle reduction of
// (min, max) pairs.  Where a block has several lanes, the even ones compute the scale of column n0 and the odd
// ones that of n0 + 8 (two or three IEEE divisions each) and they trade results.
template <int BLOCK, bool ALIGNED>
__global__ void __launch_bounds__(kThreads, 10)
quant_colwise_kernel(const __half* __restrict__ w, int K, int N, int ld, uint8_t* __restrict__ packed,
                     __half* __restrict__ scales, uint8_t* __restrict__ zps) {
  constexpr int G = BLOCK / 16;          // lanes per quantization block: 1, 2, 4, 8
  constexpr int KL = G > 4 ? G : 4;      // lanes of a warp along k
  constexpr int NL = 32 / KL;            // packed columns of a warp
  start_in_stream_order();
  const int lane = threadIdx.x & 31;
  const int kblk = blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (kblk * (16 * KL) >= K) return;     // whole warps
  const int kc = kblk * KL + lane % KL;  // chunk along k
  const int np = (blockIdx.z * kMaxGridY + blockIdx.y) * NL + lane / KL;
  if (2 * np >= N) return;               // whole warps: N / 2 is a multiple of NL
  const int na = 16 * (np / 8) + (np % 8);
  const bool has_zp = zps != nullptr;

  uint32_t va[8], vb[8];
  load_row16<ALIGNED>(w + (size_t)na * ld + kc * 16, va);
  load_row16<ALIGNED>(w + (size_t)(na + 8) * ld + kc * 16, vb);

  // (min | max << 16) of the 16 values, then of the block
  auto range16 = [](const uint32_t (&v)[8]) {
    uint32_t mn = v[0], mx = v[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
      mn = hmin2_u32(mn, v[i]);
      mx = hmax2_u32(mx, v[i]);
    }
    // pair (low halves) with (high halves)
    const uint32_t lo = __byte_perm(mn, mx, 0x5410), hi = __byte_perm(mn, mx, 0x7632);
    return __byte_perm(hmin2_u32(lo, hi), hmax2_u32(lo, hi), 0x7610);
  };
  uint32_t ra = range16(va), rb = range16(vb);
#pragma unroll
  for (int o = 1; o < G; o <<= 1) {
    const uint32_t oa = __shfl_xor_sync(0xffffffffu, ra, o), ob = __shfl_xor_sync(0xffffffffu, rb, o);
    ra = __byte_perm(hmin2_u32(ra, oa), hmax2_u32(ra, oa), 0x7610);
    rb = __byte_perm(hmin2_u32(rb, ob), hmax2_u32(rb, ob), 0x7610);
  }
  // first elements of the block, n0 | n0 + 8 (the symmetric all-zero case keeps its sign of zero)
  const uint32_t first = __shfl_sync(0xffffffffu, __byte_perm(va[0], vb[0], 0x5410), lane & ~(G - 1));

  uint32_t ma, mb;  // scale bits | zp << 16
  float rca, rcb;   // reciprocals
  auto params = [&](uint32_t range, uint32_t f, uint32_t& m, float& rc) {
    __half sc;
    uint8_t z;
    // the reference's scan starts from +-FLT_MAX, which an all-NaN block and one of infinities alone keep
    const float mn = fminf(half_bits_to_float(range & 0xffffu), __FLT_MAX__);
    const float mx = fmaxf(half_bits_to_float(range >> 16), -__FLT_MAX__);
    block_params(mn, mx, half_bits_to_float(f), has_zp, sc, z, rc);
    m = (uint32_t)__half_as_ushort(sc) | ((uint32_t)z << 16);
  };
  if constexpr (G == 1) {
    params(ra, first & 0xffffu, ma, rca);
    params(rb, first >> 16, mb, rcb);
  } else {
    const bool odd = lane & 1;
    uint32_t m;
    float rc;
    params(odd ? rb : ra, odd ? first >> 16 : first & 0xffffu, m, rc);
    const uint32_t om = __shfl_xor_sync(0xffffffffu, m, 1);
    const float orc = __shfl_xor_sync(0xffffffffu, rc, 1);
    ma = odd ? om : m;
    mb = odd ? m : om;
    rca = odd ? orc : rc;
    rcb = odd ? rc : orc;
  }

  const float za = -(float)(ma >> 16), zb = -(float)(mb >> 16);
  const unsigned long long ra2 = pack_f32x2(-rca, -rca), za2 = pack_f32x2(za, za);
  const unsigned long long rb2 = pack_f32x2(-rcb, -rcb), zb2 = pack_f32x2(zb, zb);
  uint32_t out[4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
    out[r] = assemble_word(quantize_pair<4>(va[r], ra2, za2), quantize_pair<8>(va[r + 4], ra2, za2),
                           quantize_pair<4>(vb[r], rb2, zb2), quantize_pair<8>(vb[r + 4], rb2, zb2));
  *reinterpret_cast<uint4*>(packed + (size_t)np * K + kc * 16) = make_uint4(out[0], out[1], out[2], out[3]);
  if (lane % G == 0) {
    // meta row-major [K / BLOCK, N] (reference dev_prepack_scales, column-wise branch)
    const size_t g = (size_t)((kc * 16) / BLOCK) * N + na;
    scales[g] = __ushort_as_half((unsigned short)ma);
    scales[g + 8] = __ushort_as_half((unsigned short)mb);
    if (has_zp) {
      zps[g] = (uint8_t)(ma >> 16);
      zps[g + 8] = (uint8_t)(mb >> 16);
    }
  }
}

// ---- row-wise blocks ----------------------------------------------------------------------------------
// A block is BLOCK consecutive columns at one k, i.e. one value of each column of one to eight warps.  Each warp
// reduces its 16 columns (the min / max of eight k pairs across the eight lanes of a k chunk, halving the pairs a
// lane carries at every exchange), the CTA's four warps (64 k x 64 columns; eight for blocks of 128) meet in shared memory,
// one thread per block computes the scale, and every thread picks up the parameters of its 16 k.  The weights stay in registers.
// (Measured, 11008 x 4096, block 32, symmetric: 82 us with the whole tile staged in shared memory and scanned in
// four passes.)
template <int BLOCK>
constexpr int kRowWarps = BLOCK == 128 ? 8 : 4;  // 16 columns each: whole blocks
// Word of shared memory of the parameter of row k: 16 rows and a gap of four words, so that the four k chunks whose
// parameters a warp reads 16 bytes at a time lie on different banks
__device__ __forceinline__ int param_word(int k) { return k + (k >> 4) * 4; }
template <int BLOCK, bool ALIGNED>
__global__ void __launch_bounds__(32 * kRowWarps<BLOCK>, (kRowWarps<BLOCK> == 4 ? 10 : 5))
quant_rowwise_kernel(const __half* __restrict__ w, int K, int N, int ld, uint8_t* __restrict__ packed,
                     __half* __restrict__ scales, uint8_t* __restrict__ zps) {
  constexpr int GROUPS = BLOCK / 16;          // 16-column groups (warps) per block
  constexpr int W = kRowWarps<BLOCK>;
  constexpr int NB = 16 * W / BLOCK;          // blocks per k in the tile
  __shared__ uint2 s_range[W][32];       // [16-column group][k pair] min2, max2
  __shared__ __align__(16) unsigned short s_first[W][64];  // [group][k] the group's first column
  __shared__ __align__(16) float s_recip[NB][80];  // -1 / scale
  __shared__ __align__(16) float s_zp[NB][80];     // -zero point

  start_in_stream_order();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kl = lane & 3, npl = lane >> 2;   // chunk along k, packed column of the group
  const int k0 = blockIdx.x * 64, n0 = (blockIdx.z * kMaxGridY + blockIdx.y) * (16 * W);
  const bool valid = n0 + warp * 16 < N;      // whole warps; N is a multiple of 16
  const bool has_zp = zps != nullptr;
  uint32_t va[8], vb[8];
  if (valid) {
    const __half* src = w + (size_t)(n0 + warp * 16 + npl) * ld + k0 + kl * 16;
    load_row16<ALIGNED>(src, va);
    load_row16<ALIGNED>(src + (size_t)8 * ld, vb);
    uint32_t mn[8], mx[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      mn[i] = hmin2_u32(va[i], vb[i]);
      mx[i] = hmax2_u32(va[i], vb[i]);
    }
    // exchange across the eight packed columns: lanes with the bit set keep the upper half of the pairs
#pragma unroll
    for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
      const bool upper = lane & o;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const uint32_t rmn = __shfl_xor_sync(0xffffffffu, upper ? mn[i] : mn[i + h], o);
        const uint32_t rmx = __shfl_xor_sync(0xffffffffu, upper ? mx[i] : mx[i + h], o);
        mn[i] = hmin2_u32(upper ? mn[i + h] : mn[i], rmn);
        mx[i] = hmax2_u32(upper ? mx[i + h] : mx[i], rmx);
      }
    }
    // this lane's pair: bits 4, 3, 2 of the lane select it
    const int pair = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    s_range[warp][kl * 8 + pair] = make_uint2(mn[0], mx[0]);
    if (npl == 0) {
      uint4* f = reinterpret_cast<uint4*>(&s_first[warp][kl * 16]);
      f[0] = make_uint4(va[0], va[1], va[2], va[3]);
      f[1] = make_uint4(va[4], va[5], va[6], va[7]);
    }
  }
  __syncthreads();

  // ---- one thread per quantization block ----
  for (int b = threadIdx.x; b < 64 * NB; b += 32 * W) {
    const int nb = b >> 6, k = b & 63;
    if (n0 + nb * BLOCK >= N) break;
    const int sh = (k & 1) * 16;
    float mn = __FLT_MAX__, mx = -__FLT_MAX__;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      const uint2 r = s_range[nb * GROUPS + g][k >> 1];
      mn = fminf(mn, half_bits_to_float((r.x >> sh) & 0xffffu));
      mx = fmaxf(mx, half_bits_to_float((r.y >> sh) & 0xffffu));
    }
    __half sc;
    uint8_t z;
    float rc;
    block_params(mn, mx, half_bits_to_float(s_first[nb * GROUPS][k]), has_zp, sc, z, rc);
    s_recip[nb][param_word(k)] = -rc;
    s_zp[nb][param_word(k)] = -(float)z;
    // meta column-major [K, N / BLOCK], every 16 rows permuted (reference dev_prepack_scales, :457-547): source row
    // 2t + u + 8h goes to 4t + u + 2h (scales) and 4t + 2u + h (zero points)
    const int g16 = k & ~15, u = k & 1, t = (k >> 1) & 3, h = (k >> 3) & 1;
    const size_t col = (size_t)(n0 / BLOCK + nb) * K + k0 + g16 + 4 * t;
    scales[col + u + 2 * h] = sc;
    if (has_zp) zps[col + 2 * u + h] = z;
  }
  __syncthreads();

  if (!valid) return;
  const int nb = warp / GROUPS;
  // (r, r') of the k pairs of this chunk: pair 2i, 2i + 1 in one 16-byte read
  unsigned long long r2[8], z2[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 r = *reinterpret_cast<const float4*>(&s_recip[nb][param_word(kl * 16) + 4 * i]);
    const float4 z = *reinterpret_cast<const float4*>(&s_zp[nb][param_word(kl * 16) + 4 * i]);
    r2[2 * i] = pack_f32x2(r.x, r.y);
    r2[2 * i + 1] = pack_f32x2(r.z, r.w);
    z2[2 * i] = pack_f32x2(z.x, z.y);
    z2[2 * i + 1] = pack_f32x2(z.z, z.w);
  }
  uint32_t out[4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
    out[r] = assemble_word(quantize_pair<4>(va[r], r2[r], z2[r]), quantize_pair<8>(va[r + 4], r2[r + 4], z2[r + 4]),
                           quantize_pair<4>(vb[r], r2[r], z2[r]), quantize_pair<8>(vb[r + 4], r2[r + 4], z2[r + 4]));
  *reinterpret_cast<uint4*>(packed + (size_t)(n0 / 2 + warp * 8 + npl) * K + k0 + kl * 16) =
      make_uint4(out[0], out[1], out[2], out[3]);
}

template <int BLOCK, bool ALIGNED>
cudaError_t launch_T(bool colwise, int K, int N, int ld, cudaStream_t stream, const __half* w, uint8_t* packed,
              __half* scales, uint8_t* zp) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (colwise) {
    constexpr int KL = BLOCK == 128 ? 8 : 4;
    const unsigned kblks = K / (16 * KL), groups = N / 2 / (32 / KL);
    cfg.gridDim = dim3((kblks + kWarps - 1) / kWarps, groups < kMaxGridY ? groups : kMaxGridY, (groups + kMaxGridY - 1) / kMaxGridY);
    return cudaLaunchKernelEx(&cfg, quant_colwise_kernel<BLOCK, ALIGNED>, w, K, N, ld, packed, scales, zp);
  }
  constexpr int kCols = 16 * kRowWarps<BLOCK>;
  const unsigned tiles = (N + kCols - 1) / kCols;
  cfg.gridDim = dim3(K / 64, tiles < kMaxGridY ? tiles : kMaxGridY, (tiles + kMaxGridY - 1) / kMaxGridY);
  cfg.blockDim = dim3(2 * kCols);
  return cudaLaunchKernelEx(&cfg, quant_rowwise_kernel<BLOCK, ALIGNED>, w, K, N, ld, packed, scales, zp);
}

}  // namespace

std::string launch_quant_prepack(int block, bool colwise, int K, int N, int ld,
                                 cudaStream_t stream, const __half* w, uint8_t* packed,
                                 __half* scales, uint8_t* zp) {
  const bool aligned = (reinterpret_cast<uintptr_t>(w) % 16 == 0) && (ld % 8 == 0);
  cudaError_t e = cudaSuccess;
#define BLKQ4_CASE(B)                                                                         \
  case B:                                                                                     \
    e = aligned ? launch_T<B, true>(colwise, K, N, ld, stream, w, packed, scales, zp)         \
                : launch_T<B, false>(colwise, K, N, ld, stream, w, packed, scales, zp);       \
    break;
  switch (block) {
    BLKQ4_CASE(16)
    BLKQ4_CASE(32)
    BLKQ4_CASE(64)
    BLKQ4_CASE(128)
    default:
      return "Unsupported block size: " + std::to_string(block);
  }
#undef BLKQ4_CASE
  const cudaError_t last = cudaGetLastError();
  if (e == cudaSuccess) e = last;
  if (e != cudaSuccess) return std::string("Kernel launch failed: ") + cudaGetErrorString(e);
  return std::string();
}

}  // namespace blkq4
