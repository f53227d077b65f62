// Chunk-delayed transposing kernels with the ring in tensor memory,
// half-bandwidth 5, windows of 8 samples.
#include "tring_impl.cuh"

namespace dsmvc_gb {

int launch_tring_hb5_w8(const dev::StreamJob *jobs, int count, int blocks, int per_lane, RingLayout layout,
                       dev::Sample in, dev::Sample out, RingAhead ahead, void *stream) {
    return per_lane == 2 ? rlaunch<5, 8, 2>(jobs, count, blocks, in, out, layout, ahead, stream)
                         : rlaunch<5, 8, 1>(jobs, count, blocks, in, out, layout, ahead, stream);
}

} // namespace dsmvc_gb
