// Tensor maps of TMA copies, encoded by the driver's function (looked up once, so that nothing links against the driver's library).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

extern void dl_set_error(const char* fmt, ...);

typedef CUresult (*DlEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// `rank` dimensions, the innermost (contiguous) one first; strides: bytes, of the others.  What a box holds beyond the dimensions is filled with zeros.
static int dl_tensor_map(const char* who, CUtensorMap* m, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
                         const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
    static DlEncodeTiled enc = nullptr;
    if (enc == nullptr) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || fn == nullptr) {
            dl_set_error("%s: cuTensorMapEncodeTiled not available", who);
            return -1;
        }
        enc = (DlEncodeTiled)fn;
    }
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    const CUresult r = enc(m, type, (cuuint32_t)rank, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { dl_set_error("%s: cuTensorMapEncodeTiled failed (%d)", who, (int)r); return -1; }
    return 0;
}
