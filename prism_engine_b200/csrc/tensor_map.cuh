// Host side of the kernels that copy by TMA and of those that run as clusters: tensor maps over rows of 16-bit values, and how
// many clusters are resident at once.
#pragma once

#include <cuda.h>

#include <algorithm>

#include "common.cuh"

namespace prism {

// Map of `rows` rows of `cols` 16-bit values, `pitch` values apart, in boxes of box_cols x box_rows; past the end reads zeros.
inline int encode_tensor_map(prism_cuda_ctx *ctx, CUtensorMap *map, CUtensorMapDataType type, const void *p, uint64_t cols, uint64_t rows, uint64_t pitch,
                             uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
    typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                               const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode enc = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &st) != cudaSuccess || st != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<Encode>(f);
    }();
    if (!enc) return fail(ctx, PRISM_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {pitch * 2};
    const cuuint32_t box[2] = {box_cols, box_rows}, estr[2] = {1, 1};
    const CUresult rc = enc(map, type, 2, const_cast<void *>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return rc == CUDA_SUCCESS ? PRISM_OK : fail(ctx, PRISM_E_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)rc));
}

// Clusters of `ctas` CTAs of a kernel that the GPU holds at once; 0 where it holds none (a GPC with too few SMs).
template <typename K>
inline int resident_clusters(K kernel, uint32_t ctas, uint32_t threads, size_t smem, uint32_t grid) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess) return n;
    (void)cudaGetLastError();
    return 0;
}

}  // namespace prism
