// Two-pass transposing kernels for half-bandwidth 11 (see tsolve_impl.cuh);
// one translation unit per half-bandwidth.
#include "tsolve_impl.cuh"

namespace dsmvc_gb {

int launch_tsolve_hb11(const dev::StreamJob *jobs, int count, int blocks, int threads, dev::Sample in,
                       dev::Sample out, int record_floats, void *stream) {
    return xlaunch_hb<11>(jobs, count, blocks, threads, in, out, record_floats, static_cast<cudaStream_t>(stream));
}

} // namespace dsmvc_gb
