// norm_form.h - how RMSNorm backward is cut up (norm_kernels.cuh): host arithmetic on sizes alone.
#pragma once

namespace cai {

constexpr int kNormFusedCols = 1024;   // columns one warp covers: 32 lanes x 4 chunks x 8 elements
constexpr int kNormFusedMaxH = 8192;

// The most rows of partial sums.
inline int rmsnorm_most_parts(int rows, int sms) { return rows < 2 * sms ? rows : 2 * sms; }
// Rows of partial sums that the one-sweep form writes.
inline int rmsnorm_fused_row_warps(int H) {
    const int R = (H + kNormFusedCols - 1) / kNormFusedCols;
    return R <= 1 ? 1 : R <= 2 ? 2 : R <= 4 ? 4 : 8;         // a divisor of the CTA's eight warps
}
inline int rmsnorm_fused_parts(int rows, int H, int parts_cap, int sms) {
    const int groups = 8 / rmsnorm_fused_row_warps(H);
    const long long want = (static_cast<long long>(rows) + groups - 1) / groups;
    int grid = static_cast<int>(want < 2LL * sms ? want : 2LL * sms);
    if (grid > parts_cap) grid = parts_cap;
    return grid < 1 ? 1 : grid;
}
// The rows that the form whose sums wait writes; 0 where there is no such form.
inline int rmsnorm_partial_rows(int rows, int H, int sms) {
    return rows <= 0 || H <= 0 || (H & 7) || H > kNormFusedMaxH ? 0 : rmsnorm_fused_parts(rows, H, rmsnorm_most_parts(rows, sms), sms);
}

}  // namespace cai
