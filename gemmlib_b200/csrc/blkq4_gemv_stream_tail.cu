// Decode kernel where K is not whole groups of steps for every warp, and for blocks of 32 and 16: see blkq4_gemv_stream.cuh.
#include "blkq4_gemv_stream.cuh"

namespace blkq4 {
namespace stream {

std::string launch_stream_tail(int bs, const StreamLaunch& l) {
  return bs == 0 ? launch_stream<0, false, false, true>(l) : bs == 1 ? launch_stream<1, false, false, true>(l)
       : bs == -1 ? launch_stream<-1, false, false, true>(l) : launch_stream<-2, false, false, true>(l);
}

}  // namespace stream
}  // namespace blkq4
