// Tensor maps of row-major bf16 matrices for cp.async.bulk.tensor: boxes of 64 columns in the 128-byte swizzle.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

namespace bw {
namespace lm {

constexpr int kMapCols = 64;   // columns of a box: one 128-byte swizzle atom

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// The driver's tensor-map encoder, looked up through the runtime so that the library carries no link-time dependency on libcuda (it
// must load on machines without a driver).
inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// Matrix [rows][cols], row stride ld elements (a multiple of 8), boxes of box_rows x 64 columns.
inline bool make_map(CUtensorMap* m, const void* base, int cols, long rows, long ld, int box_rows) {
    if (!encode_fn()) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kMapCols, (cuuint32_t)box_rows}, es[2] = {1, 1};
    return encode_fn()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace lm
}  // namespace bw
