// Two-pass transposing kernels with the ring in tensor memory,
// half-bandwidth 1, windows of 16 samples.
#include "xring_impl.cuh"

namespace dsmvc_gb {

int launch_xring_hb1_w16(const dev::StreamJob *jobs, int count, int blocks, int per_lane, bool tiled,
                       dev::Sample in, dev::Sample out, RingAhead ahead, void *stream) {
    return per_lane == 2 ? xrlaunch<1, 16, 2>(jobs, count, blocks, in, out, tiled, ahead, stream)
                         : xrlaunch<1, 16, 1>(jobs, count, blocks, in, out, tiled, ahead, stream);
}

} // namespace dsmvc_gb
