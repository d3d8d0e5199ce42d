// Interface of the tcgen05 Q8 GEMM kernel (q8_gemm_tc.cu).
#pragma once
#include "ops.cuh"
#include "ptx.cuh"

namespace logos {
logos_status_t launch_q8_gemm_tc(const GemmArgs& g, cudaStream_t st);
// K splits of a stand-alone product of more than 64 tokens, whose fold is a launch: what makes the kernel's own plan and the
// fold cheapest together, by the plans' costs.  gemm_pick_splits counts units of 64 tokens, a form that many tokens do not
// run in.  At most 64 MB of partial sums; one split where every SM has a row tile.  35 drawn shapes of 65 to 3411 tokens: 1 %
// slower than the best count in the mean, by that rule 6.4 % (bf16 389 x 2048 x 16512 81.8 -> 60.4 us, 256 x 3584 x 18944 95.6 ->
// 74.5, f32 173 x 2304 x 6016 24.8 -> 19.7).
int gemm_many_splits(int64_t m, int64_t n, int64_t k, int device);
logos_status_t launch_splitk_reduce(const float* partials, int splits, void* c, int c_dtype, ActOut c_act,
                                    int64_t ldc, const void* aux, int64_t m, int64_t n, int epilogue,
                                    cudaStream_t st);
// Encoded 2-D tensor maps [d1][d0], cached by (address, shape, box, swizzle).
logos_status_t cached_map(CUtensorMap* out, const void* base, CUtensorMapDataType dt, uint32_t elem, uint64_t d0,
                          uint64_t d1, uint64_t pitch1, uint32_t box0, uint32_t box1,
                          CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B);
}  // namespace logos
