// Tensor maps, the copies that use them, and shared-memory descriptors of MN-major operands, shared by the TMA-fed kernels.
// No copy here carries a cluster multicast qualifier, and every map covers this GPU's own memory only.
#pragma once

#include <cuda.h>

#include "gemm_tc.cuh"

namespace vdnn {
namespace tma {

constexpr int BOX_PIXELS = 32;
constexpr int BOX_BYTES = BOX_PIXELS * tc::BK * 4;   // 4 KB: four swizzle atoms

__device__ __forceinline__ void tma_load_rows(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int row) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(row) : "memory");
}

// Shared-memory descriptor of an MN-major tf32 operand made of 32-wide strips.  32-bit operands can only be read
// MN-major in the "128-byte swizzle with 32-byte atoms" layout: rows of 128 bytes (one pixel, 32 channels) whose
// 32-byte quarters are XORed with the row number modulo 4, the pattern repeating every 4 rows (512 bytes); the TMA
// unit writes exactly that with CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B.  One MMA takes 8 pixels = two such groups, 512
// bytes apart (stride dimension); strips of 32 rows / columns (one TMA box each) follow each other at BOX_BYTES
// (leading dimension).  Descriptor version 1, layout type 1.
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t saddr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(BOX_BYTES >> 4) << 16;
    d |= static_cast<uint64_t>(512 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(1) << 61;
    return d;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled from the driver the runtime is bound to (the library links no libcuda stub).
inline EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}

// fp32 matrix of `rows` rows of `cols` contiguous elements, row_pitch elements apart, with boxes of box_cols x box_rows.
inline int make_matrix_map(CUtensorMap* map, const float* base, size_t cols, size_t rows, size_t row_pitch, int box_cols, int box_rows,
                           CUtensorMapSwizzle swizzle) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return VDNN_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {row_pitch * sizeof(float)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1u, 1u};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? VDNN_OK : VDNN_ERR_CUDA;
}

}  // namespace tma
}  // namespace vdnn
