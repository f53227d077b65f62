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

// One-axis passes over a Float32 plane: `job.map` of columns of `size`
// samples, `job.in_elem` apart, boxes of 32 samples of 32 * `per_lane`
// columns; `job.out_map` of rows of `size` samples, `job.out_vec` apart, boxes
// of 32 samples of 32 * `per_lane` rows.
void map_input_columns(dev::StreamJob &job, int size, int per_lane);
void map_output_rows(dev::StreamJob &job, int size, int per_lane);

} // namespace dsmvc_gb
