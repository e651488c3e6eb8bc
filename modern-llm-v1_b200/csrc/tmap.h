// Host-side construction of TMA tensor maps.  The driver entry point is looked
// up at run time through the CUDA runtime, so the library has no link-time
// dependency on libcuda and still loads on a machine without a driver.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200attn {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (fn) return fn;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || p == nullptr) return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
    return fn;
}

// BF16 tensor seen as 4-D (d, t, h, b) with element strides; box = (64, box_rows, 1, 1),
// 128-byte swizzle, zero fill out of bounds.  Returns false on any driver error.
inline bool make_tmap_bf16_4d(CUtensorMap* out, const void* base, int D, int T, int H, int B, long long stride_t,
                              long long stride_h, long long stride_b, int box_rows) {
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)T, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)stride_t * 2, (cuuint64_t)stride_h * 2, (cuuint64_t)stride_b * 2};
    cuuint32_t box[4] = {64u, (cuuint32_t)box_rows, 1u, 1u};
    cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
    auto encode = [&] {
        return enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = encode();
    if (r == CUDA_ERROR_INVALID_CONTEXT) {
        // a host thread whose first CUDA call this is: the driver call, unlike the runtime's, binds no context by itself
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) return false;
        r = encode();
    }
    return r == CUDA_SUCCESS;
}

}  // namespace b200attn
