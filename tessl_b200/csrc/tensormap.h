// Tensor maps for TMA copies: the driver's encoder, looked up through the runtime (no link against libcuda), and the
// one form the kernels here use (dense tiles, no interleave, zero fill past the edges).
#pragma once
#include <cuda.h>

#include "runtime.h"

namespace tessl {

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline Result tensormap_encoder(TesslRuntime *rt, const char *what, EncodeTiled *out)
{
    if (!rt->tensormap_encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) {
            cudaGetLastError();
            return fmt("%s: the driver does not export cuTensorMapEncodeTiled", what);
        }
        rt->tensormap_encode = fn;
    }
    *out = reinterpret_cast<EncodeTiled>(rt->tensormap_encode);
    return ok();
}

/// `dims` from the innermost one; `strides` in bytes, of every dimension but the innermost.
template <int RANK>
Result make_map(EncodeTiled enc, const char *what, CUtensorMap *map, CUtensorMapDataType dt, const void *ptr,
                const cuuint64_t (&dims)[RANK], const cuuint64_t (&strides)[RANK - 1], const cuuint32_t (&box)[RANK],
                CUtensorMapSwizzle swz)
{
    cuuint32_t estr[RANK];
    for (int i = 0; i < RANK; ++i) estr[i] = 1;
    const CUresult r = enc(map, dt, RANK, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fmt("%s: cuTensorMapEncodeTiled failed (%d)", what, (int)r);
    return ok();
}

}  // namespace tessl
