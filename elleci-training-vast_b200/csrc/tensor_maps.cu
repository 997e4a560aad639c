// Tensor maps of the tensor-core kernels and the shapes they take (host code).
#include <cuda.h>

#include "common.cuh"

namespace el {

enum { MODE_FWD = 0, MODE_DX = 1, MODE_DW = 2 };

namespace tc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    // resolved once; a function-local static is initialised under the language's own lock
    static const EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(ptr);
        return nullptr;
    }();
    return fn;
}

// 2-D byte tensor [rows, cols] with row pitch `pitch`; box [box_rows, box_cols], swizzled by 128 or 32 bytes or not (0); out-of-range reads give zero.
int make_map(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch, uint32_t box_cols,
             uint32_t box_rows, int swizzle_bytes) {
    EncodeTiledFn fn = get_encode_fn();
    if (fn == nullptr) return EL_ERR_DRIVER;
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (pitch & 15) != 0) return EL_ERR_ALIGNMENT;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {pitch};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapSwizzle swizzle = swizzle_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                       : swizzle_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? EL_OK : EL_ERR_DRIVER;
}

// Output tensor [rows, cols] of 2- or 4-byte elements for the epilogue's TMA stores: boxes of `box_cols` columns x 32
// rows whose rows are 64 or 128 bytes (swizzled by that width); the store clips at the edges.
int make_map_out(CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch_bytes, int esz, int box_cols) {
    EncodeTiledFn fn = get_encode_fn();
    if (fn == nullptr) return EL_ERR_DRIVER;
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (pitch_bytes & 15) != 0) return EL_ERR_ALIGNMENT;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {pitch_bytes};
    if (box_cols * esz != 64 && box_cols * esz != 128) return EL_ERR_INVALID_ARG;
    cuuint32_t box[2] = {(cuuint32_t)box_cols, 32};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, esz == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base),
                    dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    box_cols * esz == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? EL_OK : EL_ERR_DRIVER;
}

}  // namespace tc

// EL_OK if the tensor-core kernels take the problem: 16-byte aligned operands and pitches.
int gemm_tc_eligible(int mode, const void* A, const void* B, int R, int C, int D) {
    if (R <= 0 || C <= 0 || D <= 0) return EL_ERR_UNSUPPORTED_SHAPE;
    if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return EL_ERR_ALIGNMENT;
    switch (mode) {
        case MODE_FWD: return (D % 64 == 0) ? EL_OK : EL_ERR_UNSUPPORTED_SHAPE;                    // Xq pitch D, W pitch D/4
        case MODE_DX: return (D % 16 == 0 && C % 64 == 0) ? EL_OK : EL_ERR_UNSUPPORTED_SHAPE;     // dYq pitch D(=N), W pitch C/4
        case MODE_DW: return (R % 16 == 0 && C % 16 == 0) ? EL_OK : EL_ERR_UNSUPPORTED_SHAPE;     // Gq pitch R(=N), Xq pitch C
        default: return EL_ERR_INVALID_ARG;
    }
}

}  // namespace el
