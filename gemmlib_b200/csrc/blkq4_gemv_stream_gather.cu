// Decode kernel with the fused all-gather: see blkq4_gemv_stream.cuh.
#include "blkq4_gemv_stream.cuh"

namespace blkq4 {
namespace stream {

std::string launch_stream_gather(int bs, const StreamLaunch& l) {
  return bs == 0 ? launch_stream<0, true, false, false>(l) : launch_stream<1, true, false, false>(l);
}

}  // namespace stream
}  // namespace blkq4
