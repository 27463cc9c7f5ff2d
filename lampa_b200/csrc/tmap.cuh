// Tiled TMA copies: tensor maps of row-major matrices, and the copy of one box.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"

namespace lampa {

// 2-D tiled TMA load of one box into shared memory, completion on an mbarrier; x = innermost coordinate
// (elements; x * element size must be a multiple of 16 bytes), y = row.  Single CTA, no multicast.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int32_t x, int32_t y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 :: "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
// one box from shared memory (inside the tensor: x, y >= 0), part of the bulk group of the issuing thread
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int32_t x, int32_t y, const void* src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];\n"
                 :: "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(src)) : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int32_t x, int32_t y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];\n"
                 :: "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y) : "memory");
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda)
inline PFN_cuTensorMapEncodeTiled tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(p);
    }();
    return fn;
}

// [rows][cols] tensor, row pitch = cols elements, box of box_rows x box_cols
inline bool make_map(CUtensorMap* m, const void* base, int dt, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows, bool swizzle) {
    PFN_cuTensorMapEncodeTiled enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * (cuuint64_t)dtype_bytes(dt)};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUtensorMapDataType type = dt == LAMPA_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : dt == LAMPA_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                                                                                 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    return enc(m, type, 2, const_cast<void*>(base),
               dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace lampa
