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
  // Two CTAs per SM (this launch's and the next one's) share 227 KB.  Where they fit, rings of two groups are enough from 4096 k on:
  // with four, the first copies of all CTAs, 19 MB, stand before the activations, which everything waits for.  Measured on B200, four
  // groups / two, us, block 64 with zero points: M = 1: 7168 x 4096 6.2 / 5.7, 11008 x 4096 8.5 / 8.0, 4096 x 11008 7.9 / 7.7, 8192 x 28672
  // 27.4 / 27.2; M = 4: 4096 x 11008 9.2 / 8.9; M = 8: 4096 x 4096 6.8 / 6.4, 4096 x 11008 10.8 / 10.2; two decoder blocks of 4096 and 11008
  // as one graph, M = 1, 79.8 / 75.8 (three groups 77.7; five and six as four).  2048 x 2048, M = 1, block 128 2.36 / 2.42: four there.
  // A CTA alone on its SM takes four: 11008 x 4096, M = 4 11.8 / 12.5; 8192 x 28672, M = 8, symmetric 33.4 / 36.1.
  constexpr size_t kHalfSm = (size_t)(227 * 1024) / 2 - 1024, kWholeSm = (size_t)227 * 1024;
  const size_t smem4 = stream_smem_bytes(M, K, zp_as, 4, bs), smem2 = stream_smem_bytes(M, K, zp_as, 2, bs);
  if (smem2 > kWholeSm) return kStreamUnsupported;
  const bool two_groups = smem2 <= kHalfSm ? K >= 4096 || smem4 > kHalfSm : smem4 > kWholeSm;
  StreamLaunch l{};
  StreamParams& p = l.p;
  l.ring = two_groups ? 2 : 4;
  l.smem = two_groups ? smem2 : smem4;
  p.a = a; p.out = out; p.bias = bias; p.packed = packed; p.scales = scales; p.zp = zp;
  p.M = M; p.N = N; p.K = K;
  p.tiles = N / 16;
  p.steps = K / 64;
  p.a_pitch = K + a_padding(bs);
  if (gt) p.gt = *gt;
  if (grp) {
    p.grp = *grp;
    p.tiles = grp->tile_end[grp->count - 1];
  }
  const int sms = sm_count();
  // One CTA per SM leaves the second CTA slot of every SM to the next launch (its weights stream in
  // while this launch computes).  Two per SM double the warps that compute; worth it only when the
  // tiles then still divide evenly enough.
  int grid = p.tiles < sms ? p.tiles : sms;
  if (!gt && l.smem <= kHalfSm && p.tiles > sms) {  // gather mode: one CTA per SM, so that the whole grid is resident while it waits
    const int per2 = (p.tiles + 2 * sms - 1) / (2 * sms);
    const double eff2 = (double)p.tiles / (2.0 * sms) / per2;
    if (eff2 >= 0.85) grid = p.tiles < 2 * sms ? p.tiles : 2 * sms;
  }
  l.grid = grid;
  l.one_by_one = M == 1 || (M == 2 && K >= 8192);
  l.zp = zp_as;
  l.stream = stream;
  l.early = (flags & BLKQ4_GEMM_EARLY_WEIGHT_FETCH) != 0;
  if (gt) return launch_stream_gather(bs, l);
  if (grp) return bs == 0 ? launch_stream<0, false, true, false>(l) : launch_stream<1, false, true, false>(l);
  if (tail || bs < 0) return launch_stream_tail(bs, l);
  return bs == 0 ? launch_stream<0, false, false, false>(l) : launch_stream<1, false, false, false>(l);
}

}  // namespace blkq4
