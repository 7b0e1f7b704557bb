// Host entry points of umma_gemm.cu, for the other translation units of the library.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace rmlk {

namespace tc {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn();  // matmul_tc.cu: the driver's tensor-map encoder, NULL if the driver has none
}  // namespace tc
bool tc_enabled();

// C[m, n] = A[m, k] x B[k, n], row-major f16, fp32 accumulation, one rounding.
bool umma_f16_eligible(int64_t m, int64_t n, int64_t k, const void* a, const void* b);
int umma_f16(cudaStream_t st, int64_t m, int64_t n, int64_t k, const void* a, const void* b, void* c, int* status);

}  // namespace rmlk
