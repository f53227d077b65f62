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

} // namespace

void map_input(dev::StreamJob &job, dev::Sample sample, int size, int tile_vectors, int per_lane) {
    static_assert(sizeof(CUtensorMap) == sizeof(job.map));
    job.mapped = 0;
    const std::uint64_t es = sample == dev::Sample::u8 ? 1 : sample == dev::Sample::u16 ? 2 : 4;
    const auto stride = static_cast<std::uint64_t>(job.in_vec) * es;
    if (reinterpret_cast<std::uintptr_t>(job.in) % 16 || stride % 16 || job.vectors <= 0) return;
    const bool tiled = tile_vectors > 0;
    const cuuint64_t dims[3] = {tiled ? 32U : static_cast<cuuint64_t>(size),
                                static_cast<cuuint64_t>(tiled ? tile_vectors : job.vectors),
                                tiled ? static_cast<cuuint64_t>((size + 31) / 32) : 1U};
    const cuuint64_t strides[2] = {stride, stride * dims[1]};
    if (stride == 0 || strides[1] >= (1ULL << 40)) return;
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(128 / es), static_cast<cuuint32_t>(32 * per_lane), 1};
    const cuuint32_t steps[3] = {1, 1, 1};
    const CUtensorMapDataType type = es == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                   : es == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    alignas(64) CUtensorMap map;
    if (encoder()(&map, type, 3, const_cast<void *>(job.in), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return;                             // the lanes load their own vectors
    std::memcpy(job.map, &map, sizeof(map));
    job.mapped = tiled ? 2 : 1;
}

} // namespace dsmvc_gb
