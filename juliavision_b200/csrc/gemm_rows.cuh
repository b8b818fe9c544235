// What the two kernels for unaligned operands share (gemm_rows.cu, gemm_rows_tc.cu).
#pragma once

#include <cuda_fp16.h>

#include "internal.h"

namespace b200 {

struct GrParams {
    const __half *A, *B, *bias;
    void* out;
    int64_t lda, ldb, ldo;
    int64_t M, N, K;
    int bias_per_n, epi, b_vec;
    int64_t block0;      // TWO: the launch's first row block
    int tail;            // TWO: the second launch of the product: nothing it reads waits for the first
    int steps_per_cta;   // steps of GR_STEP columns each CTA of a cluster takes
};

// The token block gemm_rows_tc.cu takes a product with, 0: none.
int gemm_rows_tc_tokens(const b200_ctx* ctx, int64_t M, int64_t N, int64_t K);
int gemm_rows_tc_launch(b200_ctx* ctx, const GrParams& p, int tokens, bool half_out);

} // namespace b200
