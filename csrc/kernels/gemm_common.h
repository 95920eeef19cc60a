// gemm_common.h - one bf16 product as the launchers see it, whatever kernel runs it.
#pragma once

#include <cuda_runtime.h>

#include "pair_form.h"

namespace cai {

struct GemmShape {
    int M, N, K;
    int a_mn, b_mn;              // operand stored with M / N contiguous instead of K
    int epi;
    float alpha;
    void* C;
    const void* R;               // residual, or the activation output of the SwiGLU epilogue
    long long lda, ldb, ldc, ldr;
    const int* seg_counts;       // ragged slabs: see cai_gemm_bf16_seg
    int seg_rows, seg_mode, grp_seg;
    int groups;                  // products of this shape in one launch, their operands grp_a / grp_b / grp_c rows apart
    long long grp_a, grp_b, grp_c;
    int sm_limit;
};

// CTA pairs, 256-row tiles (gemm_pair.cu).
int gemm_pair(const void* A, const void* B, const GemmShape& g, cudaStream_t st);

// Two products in one launch (pair_form.h).
bool pair_two_form(const GemmShape& a, const GemmShape& b, PairTwoForm* form);
int gemm_pair_two(const void* A0, const void* B0, const GemmShape& g0, const void* A1, const void* B1, const GemmShape& g1, const PairTwoForm& form,
                  cudaStream_t st);

}  // namespace cai
