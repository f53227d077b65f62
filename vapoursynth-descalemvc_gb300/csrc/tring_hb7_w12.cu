// Chunk-delayed transposing kernels with the ring in tensor memory,
// half-bandwidth 7, windows of 12 samples.
#include "tring_impl.cuh"

namespace dsmvc_gb {

int launch_tring_hb7_w12(const dev::StreamJob *jobs, int count, int blocks, int per_lane, RingLayout layout,
                       dev::Sample in, dev::Sample out, RingAhead ahead, void *stream) {
    return per_lane == 2 ? rlaunch<7, 12, 2>(jobs, count, blocks, in, out, layout, ahead, stream)
                         : rlaunch<7, 12, 1>(jobs, count, blocks, in, out, layout, ahead, stream);
}

} // namespace dsmvc_gb
