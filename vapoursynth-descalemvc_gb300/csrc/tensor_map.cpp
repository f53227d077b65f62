// See tensor_map.hpp.
#include "tensor_map.hpp"

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <stdexcept>

namespace dsmvc_gb {
namespace {

using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                            const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                            CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

Encode encoder() {
    static const Encode fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult found{};
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                                               &found);
        if (e != cudaSuccess || found != cudaDriverEntryPointSuccess || !p)
            throw std::runtime_error("the CUDA driver offers no tensor maps");
        return reinterpret_cast<Encode>(p);
    }();
    return fn;
}

// Encodes a map of a plane in up to three dimensions; false where none exists.
bool encode(unsigned char (&to)[128], const void *base, dev::Sample sample, const cuuint64_t (&dims)[3],
            std::uint64_t stride, const cuuint32_t (&box)[3], CUtensorMapSwizzle swizzle) {
    static_assert(sizeof(CUtensorMap) == sizeof(to));
    const cuuint64_t strides[2] = {stride, stride * dims[1]};
    if (reinterpret_cast<std::uintptr_t>(base) % 16 || stride == 0 || stride % 16 || strides[1] >= (1ULL << 40))
        return false;
    const cuuint32_t steps[3] = {1, 1, 1};
    const CUtensorMapDataType type = sample == dev::Sample::u8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                   : sample == dev::Sample::u16 ? CU_TENSOR_MAP_DATA_TYPE_UINT16
                                                                : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    alignas(64) CUtensorMap map;
    if (encoder()(&map, type, 3, const_cast<void *>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    std::memcpy(to, &map, sizeof(map));
    return true;
}

} // namespace

void map_input(dev::StreamJob &job, dev::Sample sample, int size, int tile_vectors, int per_lane) {
    job.mapped = 0;
    if (job.vectors <= 0) return;
    const std::uint64_t es = sample == dev::Sample::u8 ? 1 : sample == dev::Sample::u16 ? 2 : 4;
    const bool tiled = tile_vectors > 0;
    const cuuint64_t dims[3] = {tiled ? 32U : static_cast<cuuint64_t>(size),
                                static_cast<cuuint64_t>(tiled ? tile_vectors : job.vectors),
                                tiled ? static_cast<cuuint64_t>((size + 31) / 32) : 1U};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(128 / es), static_cast<cuuint32_t>(32 * per_lane), 1};
    if (encode(job.map, job.in, sample, dims, static_cast<std::uint64_t>(job.in_vec) * es, box,
               CU_TENSOR_MAP_SWIZZLE_128B))
        job.mapped = tiled ? 2 : 1;
}

void map_input_columns(dev::StreamJob &job, int size, int per_lane) {
    job.mapped = 0;
    if (job.vectors <= 0) return;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(job.vectors), static_cast<cuuint64_t>(size), 1};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(32 * per_lane), 32, 1};
    if (encode(job.map, job.in, dev::Sample::f32, dims, static_cast<std::uint64_t>(job.in_elem) * 4, box,
               CU_TENSOR_MAP_SWIZZLE_NONE))
        job.mapped = 3;
}

void map_output_rows(dev::StreamJob &job, int size, int per_lane) {
    job.out_mapped = 0;
    if (job.vectors <= 0) return;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(size), static_cast<cuuint64_t>(job.vectors), 1};
    const cuuint32_t box[3] = {32, static_cast<cuuint32_t>(32 * per_lane), 1};
    job.out_mapped = encode(job.out_map, job.out, dev::Sample::f32, dims, static_cast<std::uint64_t>(job.out_vec) * 4,
                            box, CU_TENSOR_MAP_SWIZZLE_128B) ? 1 : 0;
}

} // namespace dsmvc_gb
