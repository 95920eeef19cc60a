// pair_form.h - the form a plain bf16 product runs in on pairs of SMs (gemm_pair.cu): host arithmetic on sizes alone, for the launchers, the executor's
// list of launches and the calibrated pricing backend.
#pragma once

#include "cai_kernels.h"

namespace cai {

constexpr int kPairRows = 256, kSplitCols = 128;      // rows of a tile; columns of one that is split along K

// The form a plain product runs in: columns of a 256-row tile, slices of K that are summed in order. A function of the shape.
struct PairForm {
    int tile_cols, slices;
};

// Which form: the smallest estimate in SM cycles on a B200 of 74 pairs. A stage of 128 k-elements takes a CTA about 1150 cycles in the
// 256-wide tile (1024 of MMA) and 850 in the 128-wide one (48 KB at 54 B / cycle; 512 of MMA); a wave of tiles adds the part of its
// epilogue that nothing hides, the split form the exchange of its partials. The split form ends where its clusters no longer
// run at once: 33 of 4 and 15 of 8 CTAs are resident where the 148 SMs sit in groups of 16 to 20 (a GPU that holds fewer takes a second
// wave there). Nothing of the device enters the rule: the order of summation follows from the shape alone, on every GPU and under
// every limit on the SMs.
// Every form at 27 counts of 256 x 128 tiles from 2 to 160 and K from 256 to 8192, both operand orders (324 products): the choice is
// within 3 % of the best form but for K = 512 in at most 8 tiles of an MN-major product (8.5 us, 4 slices 7.8). us, 256-wide /
// 128-wide / 2 / 4 slices:
//   14 tiles, K 2048  15.4 / 13.4 / 10.7 /  9.3       16 tiles  15.4 / 13.7 / 10.7 / 16.5      33 tiles  15.6 / 13.9 / 11.3 / 24.8
//   36 tiles, K 2048  15.6 / 14.0 / 20.3 / 24.8       72 tiles  16.5 / 14.6 / 30.3 / 41.2      80 tiles  16.4 / 23.1
//   16 tiles, K 512    8.8 /  7.4 /  7.9 / 13.6      135 tiles, K 2048  26.2 / 23.8            160 tiles, K 2048  26.9 / 32.7
inline double pair_tile_cycles(int K, int tile_cols) {
    const double ks = static_cast<double>((static_cast<long long>(K) + 127) / 128);
    return tile_cols == 256 ? ks * 1150.0 + 2500.0 : ks * 850.0 + 1500.0;
}
inline long long pair_tile_count(int M, int N, int tile_cols) {
    return (static_cast<long long>(M) + kPairRows - 1) / kPairRows * ((static_cast<long long>(N) + tile_cols - 1) / tile_cols);
}
constexpr long long kFormPairs = 74, kSplitTiles2 = 33, kSplitTiles4 = 15;

inline PairForm pair_form(int M, int N, int K, int groups, int epi, bool segmented) {
    constexpr long long kPairs = kFormPairs;
    const long long ks = (static_cast<long long>(K) + 127) / 128;
    const long long t256 = pair_tile_count(M, N, 256) * groups, t128 = pair_tile_count(M, N, 128) * groups;
    const double wide = static_cast<double>((t256 + kPairs - 1) / kPairs) * pair_tile_cycles(K, 256);
    const double narrow = static_cast<double>((t128 + kPairs - 1) / kPairs) * pair_tile_cycles(K, 128);
    if (epi == CAI_EPI_SWIGLU) return {256, 1};
    if (!segmented) {
        const double two = ks >= 2 && t128 <= kSplitTiles2 ? (ks + 1) / 2 * 850.0 + 4500.0 : 1e30;
        const double four = ks >= 4 && t128 <= kSplitTiles4 ? (ks + 3) / 4 * 850.0 + 4500.0 : 1e30;
        if (four < two && four < wide && four < narrow) return {kSplitCols, 4};
        if (two < wide && two < narrow) return {kSplitCols, 2};
    }
    return {wide <= narrow ? 256 : 128, 1};
}


// Two products in one launch: columns of their tiles, slices of each one's K, which of them goes first. pair_two_form says whether they can go
// together and whether that is the faster way; neither may read or write what the other writes.
struct PairShape {
    int M, N, K, epi;
};
struct PairTwoForm {
    int tile_cols, slices[2], first;
};

// The schedule of two products on `pairs` pairs, of n0 tiles of c0 cycles each and n1 of c1 <= c0 (PairTwoTiles): its length.
inline double pair_two_schedule(long long n0, double c0, long long n1, double c1, long long pairs, int* heavier, int* more_first) {
    const long long q = n0 / pairs, r = n0 % pairs;
    const double base = static_cast<double>(q) * c0;
    double best = 1e30;
    *heavier = static_cast<int>(r);
    *more_first = 0;
    for (long long m = 0; m == 0 || (r > 0 && base + c0 + static_cast<double>(m) * c1 < best); ++m) {
        const long long left = n1 - m * r > 0 ? n1 - m * r : 0;
        const double light = base + static_cast<double>((left + pairs - r - 1) / (pairs - r)) * c1;
        const double heavy = r ? base + c0 + static_cast<double>(m) * c1 : 0.0;
        const double t = light > heavy ? light : heavy;
        if (t < best) {
            best = t;
            *more_first = static_cast<int>(m);
        }
    }
    return best;
}

// Two products that do not touch each other's results (the two gradients of a linear layer) in one launch, so that the last waves of one are filled
// by the other and the chain is a launch shorter: where both are one sum along K, in persistent tiles of one width; where one is split, in clusters,
// while all of them run at once. Each keeps its own order of summation, so the results are those of two launches. Measured for 38 pairs of gradients
// (tokens, in and out features; us apart / together; bursts of 3 ms with pauses):
//   1920 1000 5456  60.0 / 44.3     1920 2728 1000  39.5 / 27.8     768 2440 5728  58.8 / 46.2      3072 2352 728  36.3 / 24.6
//   512 256 1024    12.6 / 8.7      256 288 904     12.0 / 8.1      2816 352 512   13.7 / 10.0      768 848 848    14.9 / 8.3
// Against it: products that fill the tensor cores to seven tenths by themselves run at the power limit, where idle SMs cost nothing and mixed
// tiles share less in L2 (4096 2048 8192 206.8 / 210.2, 16384 2048 2048 197.8 / 201.2), and below a gain of a fifteenth by the count of waves nothing
// is left of it (4096 2048 4096 104.1 / 107.9, 3456 1408 2944 58.0 / 59.4). Tiles of 128 columns beyond one wave are fed too slowly when every SM
// is busy (1920 1000 5456 56.0, 3456 1408 5888 98.4 in wide tiles and 133.3). Clusters beyond those that run at once make a second
// wave (1024 384 808, twice four slices, 13.8 / 14.6; 256 808 10040, four slices and one sum, 31.9 / 53.9).
inline bool pair_two_form(const PairShape& a, const PairShape& b, PairTwoForm* out) {
    const PairShape* g[2] = {&a, &b};
    PairForm f[2];
    long long narrow = 0;
    for (int i = 0; i < 2; ++i) {
        if (g[i]->epi > CAI_EPI_BF16_RESIDUAL) return false;
        f[i] = pair_form(g[i]->M, g[i]->N, g[i]->K, 1, g[i]->epi, false);
        narrow += pair_tile_count(g[i]->M, g[i]->N, kSplitCols);
    }
    if (narrow > (1ll << 30)) return false;
    *out = {};
    out->slices[0] = f[0].slices;                   // the order of each product's sums is its own form's
    out->slices[1] = f[1].slices;
    out->tile_cols = kSplitCols;
    const int most = f[0].slices > f[1].slices ? f[0].slices : f[1].slices;
    if (most > 1) {
        long long clusters = 0;
        for (int i = 0; i < 2; ++i) {
            const int per_cluster = most / f[i].slices;
            clusters += (pair_tile_count(g[i]->M, g[i]->N, kSplitCols) + per_cluster - 1) / per_cluster;
        }
        return clusters <= (most == 4 ? kSplitTiles4 : kSplitTiles2);
    }
    constexpr double kLaunch = 4000.0;              // cycles from the end of a launch to the main loop of the next
    constexpr double kPairFlops = 16384.0;          // a pair's tensor cores, a cycle
    double apart = kLaunch, flops = 0;
    for (int i = 0; i < 2; ++i) {
        apart += static_cast<double>((pair_tile_count(g[i]->M, g[i]->N, f[i].tile_cols) + kFormPairs - 1) / kFormPairs) * pair_tile_cycles(g[i]->K, f[i].tile_cols);
        flops += 2.0 * g[i]->M * g[i]->N * g[i]->K;
    }
    if (narrow > kFormPairs) out->tile_cols = 256;
    out->first = g[1]->K > g[0]->K;                 // the product of the longer tiles goes first
    const PairShape &x = *g[out->first], &y = *g[1 - out->first];
    const long long nx = pair_tile_count(x.M, x.N, out->tile_cols), ny = pair_tile_count(y.M, y.N, out->tile_cols);
    int heavier, more;
    const double together = pair_two_schedule(nx, pair_tile_cycles(x.K, out->tile_cols), ny, pair_tile_cycles(y.K, out->tile_cols),
                                              nx + ny < kFormPairs ? nx + ny : kFormPairs, &heavier, &more);
    return together <= 14.0 / 15.0 * apart && flops <= 0.7 * apart * kFormPairs * kPairFlops;
}

// Whether a gate / up projection of F features and its SwiGLU are one sum along K, and faster as one launch.
inline bool pair_swiglu_pays(int M, int F, int K) {
    if (M <= 0 || F <= 0 || K <= 0 || (F & 7) || F > (1 << 29)) return false;
    const PairForm f = pair_form(M, 2 * F, K, 1, CAI_EPI_BF16, false);
    if (f.slices > 1) return false;                 // the sums would be others
    auto cycles = [&](int cols) { return static_cast<double>((pair_tile_count(M, 2 * F, cols) + kFormPairs - 1) / kFormPairs) * pair_tile_cycles(K, cols); };
    // against the plain product: the exponentials of the last tile; a launch less, and gu and act not carried once more (three words of a feature at
    // 3.4 KB a cycle)
    return cycles(256) + 2000.0 <= cycles(f.tile_cols) + 4000.0 + 6.0 / 3400.0 * M * F;
}

}  // namespace cai
