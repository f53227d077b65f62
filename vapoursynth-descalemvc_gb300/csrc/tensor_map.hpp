// Tensor maps of the planes that the kernels with the ring in tensor memory
// read (tring_impl.cuh).
#pragma once

#include "stream.cuh"

namespace dsmvc_gb {

// Writes `job.map` and `job.mapped` for a pass over `job.vectors` vectors of
// `size` samples, adjacent samples, `job.in_vec` samples apart; `tile_vectors`
// > 0: the vectors' samples lie in tiles of 32, [sample / 32][vector][32],
// with that many vectors a tile.  A box is 128 bytes of 32 * `per_lane`
// vectors.  Planes that a tensor map cannot describe (vectors not 16-byte
// aligned) keep mapped = 0.
void map_input(dev::StreamJob &job, dev::Sample sample, int size, int tile_vectors, int per_lane);

} // namespace dsmvc_gb
