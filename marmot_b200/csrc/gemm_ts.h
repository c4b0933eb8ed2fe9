// Parameters and launchers of the tcgen05 matmul with weights in tensor memory (gemm_ts.cu).
#pragma once

#include "gemm_plan.h"
#include "kernels.h"

#include <cuda.h>

namespace mcu {

struct TsMaps {
    CUtensorMap x;               // fp16 activations [rows][kp]
    CUtensorMap w[TS_MAX_JOBS];  // packed weights of each matrix
};
// Shares of cut tiles (gemm_ts_workspace_bytes(), 0 tickets in `counters` between launches, one int per SM).
size_t gemm_ts_workspace_bytes();
bool gemm_ts_supported(int kind, const void *W, int T, int K, int F);
// up to TS_MAX_JOBS matrices of one kind that read the same activations (fp16 from launch_act_half_fused_from), in one launch
cudaError_t launch_gemm_ts(int kind, const GemvJobSpec *jobs, int n_jobs, const __half *xh, const float *rowscale, int ldxh,
                           int T, int K, float *partial, int *counters, int *err_flag, cudaStream_t s);
// stacked matrices: rows that are not 16-byte multiples need a multiple of eight rows per group
bool gemm_ts_grouped_supported(int kind, const void *W, int K, int F);
cudaError_t launch_gemm_ts_grouped(int kind, const GemvJobSpec *jobs, int n_jobs, int n_groups, const __half *xh, const float *rowscale,
                                   int ldxh, int total_rows, int K, const int *group_counts, const int *group_offsets,
                                   float *partial, int *counters, int *err_flag, cudaStream_t s);

// The same on integers for a handful of tokens (gemm_ti.cu: Q4_K, Q6_K): exact sub-block dots.  xq from
// launch_act_int_fused.
size_t gemm_ti_xq_bytes(int kind, int rows, int K);
bool gemm_ti_supported(int kind, const void *W, int K, int F);
cudaError_t launch_gemm_ti(int kind, const GemvJobSpec *jobs, int n_jobs, const uint8_t *xq, int T, int K,
                           float *partial, int *counters, int *err_flag, cudaStream_t s);
cudaError_t launch_gemm_ti_grouped(int kind, const GemvJobSpec *jobs, int n_jobs, int n_groups, const uint8_t *xq,
                                   int total_rows, int K, const int *group_counts, const int *group_offsets,
                                   float *partial, int *counters, int *err_flag, cudaStream_t s);

// host helpers of the two
bool ts_loose(int kind, const void *W, long row_bytes);
cudaError_t ts_encode(CUtensorMap *m, CUtensorMapDataType type, const void *base, cuuint64_t d0, cuuint64_t d1, cuuint64_t stride,
                      cuuint32_t b0, cuuint32_t b1, CUtensorMapSwizzle sw);
cudaError_t ts_encode_weights(int kind, CUtensorMap *m, const void *W, long row_bytes, size_t rows, bool loose);
cudaError_t ts_grouped_params(int kind, const GemvJobSpec *jobs, int n_jobs, int n_groups, int total_rows, int K,
                              const int *group_counts, const int *group_offsets, TsParams &p, TsMaps &maps);

}  // namespace mcu
