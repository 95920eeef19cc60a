// gemm_common.h - one bf16 product as the launchers see it, whatever kernel runs it.
#pragma once

#include <cuda_runtime.h>

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

// The form a plain product runs in: columns of a 256-row tile, slices of K that are summed in order. A function of the shape.
struct PairForm {
    int tile_cols, slices;
};
PairForm pair_form(int M, int N, int K, int groups, int epi, bool segmented);
// CTA pairs, 256-row tiles (gemm_pair.cu).
int gemm_pair(const void* A, const void* B, const GemmShape& g, cudaStream_t st);

// Two products in one launch: columns of their tiles, slices of each one's K, which of them goes first. pair_two_form says whether they can go
// together and whether that is the faster way; neither may read or write what the other writes.
struct PairTwoForm {
    int tile_cols, slices[2], first;
};
bool pair_two_form(const GemmShape& a, const GemmShape& b, PairTwoForm* form);
int gemm_pair_two(const void* A0, const void* B0, const GemmShape& g0, const void* A1, const void* B1, const GemmShape& g1, const PairTwoForm& form,
                  cudaStream_t st);

}  // namespace cai
