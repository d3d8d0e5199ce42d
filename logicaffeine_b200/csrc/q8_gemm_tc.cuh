// Interface of the tcgen05 Q8 GEMM kernel (q8_gemm_tc.cu).
#pragma once
#include "ops.cuh"
#include "ptx.cuh"

namespace logos {
logos_status_t launch_q8_gemm_tc(const GemmArgs& g, cudaStream_t st);
// Tokens of a unit of the wide form that a product without K splits runs in; 0: another form.
int gemm_wide_tokens(int64_t m, int64_t n, int64_t k, int device);
logos_status_t launch_splitk_reduce(const float* partials, int splits, void* c, int c_dtype, ActOut c_act,
                                    int64_t ldc, const void* aux, int64_t m, int64_t n, int epilogue, int device,
                                    cudaStream_t st);
// Encoded 2-D tensor maps [d1][d0], cached by (address, shape, box, swizzle).
logos_status_t cached_map(CUtensorMap* out, const void* base, CUtensorMapDataType dt, uint32_t elem, uint64_t d0,
                          uint64_t d1, uint64_t pitch1, uint32_t box0, uint32_t box1,
                          CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B);
}  // namespace logos
