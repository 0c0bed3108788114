// Decode kernel (blkq4_gemv_stream.cuh): which problems it takes, and with what rings and grid.
#include <cstddef>
#include <cstdint>
#include <string>

#include "blkq4_gemv_stream.cuh"
#include "ms_blkq4gemm.h"

namespace blkq4 {

using namespace stream;

namespace {

size_t stream_smem_bytes(int M, int K, Zp zp, int D, int bs) {
  const int MS = (M + 1) & ~1, PW = zp == Zp::kOwnSums ? 2 * kWarps : kWarps, steps = K / 64;
  const size_t blocks = (size_t)steps * blocks_per_step(bs);
  return (size_t)kWarps * D * slot_bytes(bs) + blocks * 64 + (zp != Zp::kNone ? blocks * 32 : 0) + (size_t)2 * PW * 16 * MS * 4 + 256 +
         (size_t)M * (K + a_padding(bs)) * 2;
}

// Blocks of 32 and 16, against the generic kernel (which scales in fp16; larger problems than these are the tensor-core kernel's, see
// gemm_tc_takes_skinny).  Every block has a sum to be scaled, with zero points a subtraction too, per eight rows, which the generic
// kernel's conversion has not: more rows and smaller blocks are its side.  Measured on B200, generic / this, us, M = 1, 2, 4, 8:
//   block 32, symmetric:   512 x 512 3.1 / 1.7, 1.8, 2.1, 2.7;  1024 x 4096 3.8 / 2.3, 2.5, 2.8, 3.4;  2048 x 2048 3.9 / 2.5, 2.6, 3.0, 3.6;
//                          2048 x 8192 7.9 / 4.3, 4.6, 5.0, 6.1;  4096 x 4096 7.0 / 4.4, 5.0, 5.9, 7.1;  5632 x 2048 7.9 / 4.5, 5.0, 6.7, 7.2
//   with zero points:      1024 x 4096 3.8 / 2.5, 2.7, 3.0, 3.6;  1984 x 3008 5.7 / 3.1, 3.3, 3.7, 4.5;  2048 x 2048 4.0 / 2.8, 3.0, 3.6, 4.4;
//                          4096 x 4096 7.1 / 5.1, 5.6, 6.6, 7.9
//   block 16, symmetric:   1024 x 4096 3.8 / 2.5, 2.7, 3.1, 3.8;  2048 x 2048 3.9 / 3.0, 3.0, 4.0, 5.4;  4096 x 4096 7.2 / 5.4, 6.2, 7.5, 8.5
//   with zero points:      1024 x 4096 4.0 / 2.8, 3.0, 3.5, 4.3;  2048 x 2048 4.1 / 3.6, 3.9, 4.8, 6.4;  4096 x 4096 7.9 / 6.6, 7.4, 8.9, 10.0;
//                          M = 2: 576 x 14720 5.8 / 6.1, 3200 x 3200 to 6656 1.15 of the generic kernel's time
// Below 512 k or columns nothing was measured: they stay on the generic kernel.
bool small_blocks_are_faster(int block, int M, int N, int K, bool has_zp) {
  if (K < 512 || N < 512) return false;
  if (block == 32) return M <= 4 || !has_zp || K < 2048;
  return has_zp ? M == 1 || (M <= 4 && K < 2048 && N <= 8192) : M <= 2 || (M <= 4 && K < 2048);
}

}  // namespace

const char* const kStreamUnsupported = "unsupported by the stream kernel";

bool gemv_stream_takes(int block, bool colwise, int M, int N, int K) {
  const int group_k = kGroupSteps * 64;
  return colwise && block >= 64 && M >= 1 && M <= 8 && K % group_k == 0 && K / group_k >= kWarps &&
         (size_t)K * N / 2 < ((size_t)1 << 40) && stream_smem_bytes(M, K, Zp::kOwnSums, 2, 0) <= (size_t)227 * 1024;  // whatever the zero points: part of the interface
}

// Returns kStreamUnsupported when the shape is outside this kernel (the caller then takes another one).
std::string launch_gemv_stream(int block, bool colwise, int M, int N, int K, cudaStream_t stream,
                               const __half* a, const uint8_t* packed, const __half* scales,
                               const uint8_t* zp, __half* out, const __half* bias, unsigned flags,
                               const GatherTable* gt, const GemmGroup* grp) {
  const int group_k = kGroupSteps * 64;
  const bool tail = K % group_k != 0 || K / group_k < kWarps;
  const int bs = block == 128 ? 1 : block == 64 ? 0 : block == 32 ? -1 : -2;
  if (bs < 0 && (gt || grp || !small_blocks_are_faster(block, M, N, K, zp != nullptr))) return kStreamUnsupported;
  if (!colwise || M < 1 || M > 8 || K % 64 != 0 || (tail && (gt || grp)) ||
      reinterpret_cast<uintptr_t>(scales) % 16 != 0 || (zp && reinterpret_cast<uintptr_t>(zp) % 16 != 0) ||
      (size_t)K * N / 2 >= ((size_t)1 << 40))
    return kStreamUnsupported;
  // M <= 2: see the kernel; a launch of several matrices decides as their own launches do
  const Zp zp_as = !zp ? Zp::kNone : M > 2 || tail || bs < 0 ? Zp::kPerStep : Zp::kOwnSums;
  // Two CTAs fit on an SM, this launch's and the next one's, if each takes less than half of its shared memory.  The grid has one CTA per
  // SM, so that the second slot is the next launch's (its weights stream in while this launch computes), or two, which
  // doubles the warps that compute: worth it only when the tiles then still divide evenly enough.  Gather mode: one, so that the
  // whole grid is resident while it waits.
  constexpr size_t kHalfSm = (size_t)(227 * 1024) / 2 - 1024, kWholeSm = (size_t)227 * 1024;
  const size_t smem4 = stream_smem_bytes(M, K, zp_as, 4, bs), smem2 = stream_smem_bytes(M, K, zp_as, 2, bs);
  if (smem2 > kWholeSm) return kStreamUnsupported;
  const int sms = sm_count(), tiles = grp ? grp->tile_end[grp->count - 1] : N / 16;
  const int rounds2 = (tiles + 2 * sms - 1) / (2 * sms);
  const bool two_per_sm = !gt && smem2 <= kHalfSm && tiles > sms && (double)tiles / (2.0 * sms) / rounds2 >= 0.85;
  // Groups in flight per warp.  With four, the first copies of all CTAs stand before the activations, which everything waits for: 19 MB where
  // there are two CTAs per SM.  Two are enough there, and where they hold a warp's whole slice of a tile (up to 4096 k); a CTA
  // alone on its SM has too little in flight with two of a longer slice.  Measured on B200, two / four groups, time ratio, M = 1 and 2 with
  // the early weight fetch: two CTAs per SM (N = 4096 and 8192) 4096 k 0.86 to 1.00, 5120 0.94 to 0.99, 8192 0.90 to 0.99, 11008 0.96 to 1.03;
  // one CTA per SM (N = 1024, 2048, 3584, 14336) 2048 to 4096 k 0.92 to 1.07, mean 0.99, 4352 1.06 to 1.21, 8192 1.00 to 1.25, 11008 1.12 to
  // 1.26 (1 x 11008 x 14336 27.3 / 24.1 us); short last groups of one CTA per SM: 2112 1.0 to 1.1, 4160 and 5696 1.0 to 1.15.  In gather mode:
  // 4096 k 0.97 to 1.00, 5120 x 1728 1.08, 8192 x 14336 1.11.
  // Two decoder blocks of 4096 and 11008 as one graph, M = 1, four / two groups 79.8 / 75.8 us (three groups 77.7; five and six as four).
  // Where two CTAs fit with rings of two only, those are taken; a CTA that is alone on its SM in any case takes four: 11008 x 4096, M = 4
  // 11.8 / 12.5; 8192 x 28672, M = 8, symmetric 33.4 / 36.1.
  const bool slice_fits = !tail && bs >= 0 && K <= 2 * kWarps * group_k;
  const bool two_groups = smem2 <= kHalfSm ? two_per_sm || slice_fits || smem4 > kHalfSm : smem4 > kWholeSm;
  StreamLaunch l{};
  StreamParams& p = l.p;
  l.ring = two_groups ? 2 : 4;
  l.smem = two_groups ? smem2 : smem4;
  p.a = a; p.out = out; p.bias = bias; p.packed = packed; p.scales = scales; p.zp = zp;
  p.M = M; p.N = N; p.K = K;
  p.tiles = tiles;
  p.steps = K / 64;
  p.a_pitch = K + a_padding(bs);
  if (gt) p.gt = *gt;
  if (grp) p.grp = *grp;
  l.grid = two_per_sm ? (tiles < 2 * sms ? tiles : 2 * sms) : tiles < sms ? tiles : sms;
  l.one_by_one = M == 1 || (M == 2 && (tail ? K >= 8192 : K > 3 * kWarps * group_k));
  l.zp = zp_as;
  l.stream = stream;
  l.early = (flags & BLKQ4_GEMM_EARLY_WEIGHT_FETCH) != 0;
  if (gt) return launch_stream_gather(bs, l);
  if (grp) return bs == 0 ? launch_stream<0, false, true, false>(l) : launch_stream<1, false, true, false>(l);
  if (tail || bs < 0) return launch_stream_tail(bs, l);
  return bs == 0 ? launch_stream<0, false, false, false>(l) : launch_stream<1, false, false, false>(l);
}

}  // namespace blkq4
