// moe.cuh -- shared between moe.cu and the grouped mode of qmatmul_tc.cu
#pragma once
#include "common.cuh"

namespace b200 {

// grouped-GEMM work: rows [x_row0, x_row0 + count) of the expert-sorted activations, all routed to `expert`
struct MoeChunk { int expert, x_row0, count; };

// grouped dequant-GEMM on the tcgen05 pipeline (qmatmul_tc.cu): y[sg][row_map[x_row0 + i]][j] = row_scale * sum_k xs[x_row0 + i][k] w[sg][expert * n + j][k] for nseg <= 2
// stacks w of GGML blocks [E * n, k] (row_map null: the sorted row itself).  xs: fp16 K4 [rows_padded, k] (expert-sorted); the chunk list and its length live on the
// device, chunk_rows (32, 64 or 128) is what it was cut into, max_chunks its bound
bool qmatmul_tc_moe_supported(int n, int k, int ggml_type);
void qmatmul_tc_moe(const void* xs_f16_k4, int xs_rows, int nseg, const void* const* w, int num_experts, float* const* y, int64_t ldy, int n, int k, int ggml_type,
                    const MoeChunk* chunks, const int* num_chunks, int max_chunks, int chunk_rows, const uint32_t* row_map, const float* row_scale, cudaStream_t st);

// the same with block-scaled e4m3 experts; xs fp16 in natural order, chunks of 32 rows; norm: 2 floats of device scratch
bool qmatmul_tc_moe_fp8_supported(int n, int k, int by, int bx);
void qmatmul_tc_moe_fp8(const void* xs_f16, int xs_rows, const void* w, const float* scale, int num_experts, float* y, int64_t ldy, int n, int k, int by, int bx,
                        const MoeChunk* chunks, const int* num_chunks, int max_chunks, const uint32_t* row_map, const float* row_scale, float* norm,
                        cudaStream_t st);

}  // namespace b200
