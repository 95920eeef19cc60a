// gemm_pair.cu - bf16 GEMM on CTA pairs (tcgen05 cta_group::2), the plain (single GPU) products.
//
//   C[M,N] = alpha * sum_k A(m,k) * B(n,k)   (+ epilogue)
//
// Two CTAs on neighbouring SMs (a cluster of two) compute one 256 x BN tile. Each loads its own 128 rows of A and its own
// BN / 2 rows of B into its own shared memory; the MMA, issued by one thread of the even CTA, reads both halves of B from
// both SMs. What bounds the one-CTA kernel (gemm_tcgen05.cu) is shared-memory bandwidth: a 128 x 256 x 16 MMA takes 128
// cycles and reads 12 KB (96 B / cycle) while TMA writes the next 12 KB (96 B / cycle) against 128 B / cycle per SM. The pair
// reads and writes 8 KB per SM for the same arithmetic, and L2 delivers a third less.
//
// Warp 0 feeds a ring of shared-memory stages with TMA (no multicast: every CTA loads its own part), warp 1 of the even CTA
// issues the MMAs, warps 2-9 drain the accumulator. Two accumulators per CTA in TMEM let the epilogue of a tile overlap the
// main loop of the next. The epilogue goes through shared memory and leaves by TMA: full 128-byte rows instead of 16 bytes per
// lane, edges clipped by the tensor map, the fp32 accumulation into C as a TMA reduction in L2 (one rounding and subnormals kept,
// like a load and an add); the residual is read into registers while the main loop still runs, whole rows at a time. (bf16 stores straight from the
// registers, a 32-byte sector per lane, measured the same on aligned rows and up to 20 % slower on rows of 2000 bytes.)
//
// Measured against the one-CTA kernel (L2 flushed): 8192^3 812 -> 706 us (1556 TFLOP/s), 16384 x 2048 x 16384 1062 -> 712 us,
// 16384 x 16384 x 2048 with SwiGLU 1026 -> 773 us, weight gradient 16384 x 2048 x 16384 1117 -> 794 us. One barrier round trip per
// 64 k-elements instead of 128 held it at 1430 TFLOP/s: with data present, the issuing thread spends some 300 cycles between a
// satisfied wait and its first MMA.
#include "../plan/formats.h"
#include "cai_kernels.h"
#include "gemm_common.h"
#include "host_common.h"
#include "sm100.cuh"

namespace cai {

namespace pair {
constexpr int kBM = kPairRows;           // rows of a tile (128 per CTA)
constexpr int kBK = 64;               // k-elements of a block (one 128-byte row of a K-major operand)
constexpr int kPerStage = 2;          // blocks of a stage: one barrier round trip of the issuing thread per 128 k-elements
constexpr int kUmmaK = 16;
constexpr int kThreads = 320;         // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int kEpiWarps = 8;
constexpr int kABytes = 128 * kBK * 2;
constexpr int kBox = 4096;            // an epilogue box: 32 rows x 128 bytes
template <int BN> constexpr int kBBytes = BN / 2 * kBK * 2;
template <int BN> constexpr int kBlock = kABytes + kBBytes<BN>;
template <int BN> constexpr int kStages = BN == 256 ? 3 : 4;
constexpr int kMaxSlabs = 256;        // ragged rows: slabs whose live halves a launch can count ahead
template <int BN> constexpr int kSmem = kStages<BN> * kPerStage * kBlock<BN> + kEpiWarps * kBox + 512 + (kMaxSlabs + 4) * 4 + 1024;
}  // namespace pair

struct PairParams {
    int M, N, K;
    int a_mn, b_mn;
    int epi;
    float alpha;
    int tiles_m, tiles_n, group_m, groups;
    int tile0;                    // split form: first tile of this launch
    const int* seg_counts;
    int seg_rows, seg_mode, grp_seg;
    bool overlap;                 // the next kernel of the stream may come in while this one finishes (not under a limit on the SMs)
    int grp_slabs;                // ragged rows, live halves counted ahead: slabs of a group (0: the ordinary walk)
    void* C;                      // split form: results leave through registers
    const __nv_bfloat16* R;       // residual, read row by row
    long long ldc, ldr, grp_c;    // grp_c: rows between the groups of C and R
    int* status;
};

// One product of a launch: maps of A, B, C and (SwiGLU) the activation, and what else the kernel has to know.
struct PairProduct {
    CUtensorMap map[4];
    PairParams p;
};
// A launch of one product, or of two plain ones that do not touch each other's results (see gemm_pair_two).
template <int kProducts> struct PairLaunch {
    PairProduct product[kProducts];
    int heavier, more_first;      // two products: how many pairs have one tile of the first product more than the others, and how
                                  // many tiles of the second such a pair takes
};

__host__ __device__ __forceinline__ bool pair_seg_live(const PairParams& p, int g, int row0) {
    const int slab = row0 / p.seg_rows;
    return row0 - slab * p.seg_rows < p.seg_counts[g * p.grp_seg + slab];
}
// Is the 128-row half that starts at row `row0` of group g computed and written?
__host__ __device__ __forceinline__ bool pair_half_live(const PairParams& p, int g, int row0) {
    return row0 < p.M && (p.seg_mode != 1 || pair_seg_live(p, g, row0));
}

// The k-range of one tile in stages of 128 elements: all of K, or under seg_mode 2 the live rows at the front of each slab
// (a stage lies in one slab). A step costs no division, and a count is read once per slab; asking for both blocks of every
// stage whether they are live (two divisions and two reads) kept the issuing thread some 350 cycles per stage, dead ones included.
// 64 products of 4096 x 1536, and of 3072 x 4096, over some 1024 of 2048 rows each: 1246 -> 881 and 2477 -> 1773 us.
template <bool kRagged>
struct PairStages {
    const int* counts;
    int slab_rows, slabs, slab = -1, base = 0, rows = 0, at = 0;   // at: element of the next stage inside the slab
    __device__ __forceinline__ PairStages(const PairParams& p, int g) {
        const bool ragged = kRagged && p.seg_mode == 2;
        counts = ragged ? p.seg_counts + g * p.grp_seg : nullptr;
        slab_rows = ragged ? p.seg_rows : p.K;
        slabs = ragged ? (p.K + p.seg_rows - 1) / p.seg_rows : 1;
    }
    // Next stage with data: its number and which of its two blocks hold any (bit per block).
    __device__ __forceinline__ bool next(const PairParams& p, int& ks, uint32_t& live) {
        while (at >= rows) {
            if (++slab >= slabs) return false;
            base = slab * slab_rows;
            rows = min(slab_rows, p.K - base);
            if (kRagged && counts) rows = min(rows, counts[slab]);
            at = 0;
        }
        ks = (base + at) / (pair::kPerStage * pair::kBK);
        live = rows - at > pair::kBK ? 3u : 1u;
        at += pair::kPerStage * pair::kBK;
        return true;
    }
};

__host__ __device__ __forceinline__ void pair_tile_coords(const PairParams& p, int tile_all, int& tm, int& tn, int& grp) {
    const int per_product = p.tiles_m * p.tiles_n;
    grp = tile_all / per_product;
    const int tile = tile_all - grp * per_product;
    const int per_group = p.group_m * p.tiles_n;
    const int g = tile / per_group;
    const int first_m = g * p.group_m;
    const int gsz = min(p.tiles_m - first_m, p.group_m);
    const int in = tile - g * per_group;
    tm = first_m + in % gsz;
    tn = in / gsz;
}

// The tiles of one pair of CTAs. Ragged rows are walked over live halves of 128 rows only, numbered group by group, with one that is
// not live behind an odd number of them: first[s] is 2 x the number of the first half of slab s (at the end of a group + 1 where its
// last half is not live). A tile takes two neighbouring halves of its group, of whatever slabs: each CTA of a pair loads, multiplies and
// writes its own. So every pair gets its share of the tiles, and none is half empty but the last of a group. us, tiles by their place in
// the full slabs / live tiles of each slab / live halves: 64 slabs of one group each, some 1024 of 2048 rows live, 3072 x 4096 1605 / 1351 /
// 1351; 8 groups of 8 slabs, 3072 x 4096, 128 rows full 151 / 255 / 151, 384 rows full 386 / 493 / 383, 1152 rows at random 1080 / 710 / 620.
struct PairTiles {
    int tile, stride, group = 0;
    __host__ __device__ __forceinline__ PairTiles(int pair, int pairs) : tile(pair), stride(pairs) {}
    // The next tile: its column tile, its group, the first row (inside the group) of the half of CTA `rank`, and whether that half is live.
    __host__ __device__ __forceinline__ bool next(const PairParams& p, const int* first, int rank, int& row, int& tn, int& grp, bool& live) {
        if (p.grp_slabs) {
            if (tile >= (first[p.grp_slabs * p.groups] >> 2) * p.tiles_n) return false;
            while (tile >= (first[(group + 1) * p.grp_slabs] >> 2) * p.tiles_n) ++group;
            grp = group;
            int lo = group * p.grp_slabs, hi = lo + p.grp_slabs;
            const int h0 = first[lo] >> 1, end = first[hi], rows = ((end >> 1) - h0) >> 1;
            const int at = tile - (h0 >> 1) * p.tiles_n, per_raster = p.group_m * p.tiles_n;
            const int g = at / per_raster, in = at - g * per_raster;
            const int left = rows - g * p.group_m, gsz = left < p.group_m ? left : p.group_m;
            tn = in / gsz;
            int h = h0 + 2 * (g * p.group_m + in - tn * gsz) + rank;
            live = h < (end >> 1) - (end & 1);
            if (!live) --h;                    // the other CTA's rows once more: loaded, never written
            while (hi - lo > 1) {              // its slab: the last that starts at h or before
                const int mid = (lo + hi) >> 1;
                if (first[mid] >> 1 <= h) lo = mid;
                else hi = mid;
            }
            row = (lo - group * p.grp_slabs) * p.seg_rows + (h - (first[lo] >> 1)) * 128;
            tile += stride;
            return true;
        }
        for (; tile < p.tiles_m * p.tiles_n * p.groups; tile += stride) {
            int tm;
            pair_tile_coords(p, tile, tm, tn, grp);
            row = tm * pair::kBM + rank * 128;
            live = pair_half_live(p, grp, row);
            if (live || pair_half_live(p, grp, row ^ 128)) {
                tile += stride;
                return true;
            }
        }
        return false;
    }
};
// Tiles of a launch of two products. The first, whose tiles take longer, goes round the pairs; the second fills up: the pairs that took a tile less
// take more of it. A closed form of what a list ordered by length would give, and the same on every GPU.
struct PairTwoTiles {
    int pair, pairs, round = 0, second = 0;
    __host__ __device__ __forceinline__ PairTwoTiles(int pair_, int pairs_) : pair(pair_), pairs(pairs_) {}
    // The number of the next tile inside its product; which: the product.
    __host__ __device__ __forceinline__ bool next(int tiles0, int tiles1, int heavier, int more_first, int& which, int& tile) {
        tile = pair + round * pairs;
        which = 0;
        if (tile < tiles0) {
            ++round;
            return true;
        }
        which = 1;
        if (pair < heavier) {
            tile = second * heavier + pair;
            return second++ < more_first && tile < tiles1;
        }
        tile = more_first * heavier + second * (pairs - heavier) + pair - heavier;
        ++second;
        return tile < tiles1;
    }
};
template <int kProducts, bool kRagged> struct PairWalk {
    PairTiles tiles;
    __device__ __forceinline__ PairWalk(int pair, int pairs) : tiles(pair, pairs) {}
    __device__ __forceinline__ bool next(const PairLaunch<1>& l, const int* first, int rank, int& row, int& tn, int& grp, bool& live, int& which) {
        which = 0;
        const PairParams& p = l.product[0].p;
        if (kRagged) return tiles.next(p, first, rank, row, tn, grp, live);
        if (tiles.tile >= p.tiles_m * p.tiles_n * p.groups) return false;
        int tm;
        pair_tile_coords(p, tiles.tile, tm, tn, grp);
        tiles.tile += tiles.stride;
        row = tm * pair::kBM + rank * 128;
        live = row < p.M;
        return true;
    }
};
template <> struct PairWalk<2, false> {
    PairTwoTiles tiles;
    __device__ __forceinline__ PairWalk(int pair, int pairs) : tiles(pair, pairs) {}
    __device__ __forceinline__ bool next(const PairLaunch<2>& l, const int*, int rank, int& row, int& tn, int& grp, bool& live, int& which) {
        int tile, tm;
        const PairParams &a = l.product[0].p, &b = l.product[1].p;
        if (!tiles.next(a.tiles_m * a.tiles_n, b.tiles_m * b.tiles_n, l.heavier, l.more_first, which, tile)) return false;
        pair_tile_coords(l.product[which].p, tile, tm, tn, grp);
        row = tm * pair::kBM + rank * 128;
        live = row < l.product[which].p.M;
        return true;
    }
};
__host__ __device__ __forceinline__ int pair_live_halves(const PairParams& p, int slab) {
    const int grp = slab / p.grp_slabs, in = slab - grp * p.grp_slabs;
    int n = p.seg_counts[grp * p.grp_seg + in];
    if (n > p.seg_rows) n = p.seg_rows;
    if (n > p.M - in * p.seg_rows) n = p.M - in * p.seg_rows;
    return n > 0 ? (n + 127) / 128 : 0;
}
// first[s] for s = 0 .. all slabs, by one warp.
__device__ __forceinline__ void pair_count_halves(const PairParams& p, int* first, int lane) {
    constexpr int kChunks = pair::kMaxSlabs / 32;
    const int slabs = p.grp_slabs * p.groups;
    int n[kChunks];
#pragma unroll
    for (int i = 0; i < kChunks; ++i) n[i] = i * 32 + lane < slabs ? pair_live_halves(p, i * 32 + lane) : 0;
    int before = 0;
    if (lane == 0) first[0] = 0;
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
        if (i * 32 >= slabs) break;
        // one slab a group: its odd half is added here
        const int odd = p.grp_slabs == 1 ? n[i] & 1 : 0;
        int sum = n[i] + odd;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        if (i * 32 + lane < slabs) first[i * 32 + lane + 1] = (before + sum) * 2 + odd;
        before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (p.grp_slabs == 1) return;
    // several: which groups have an odd number (so far halves are numbered without the added ones), then every slab moves by those before it
    __syncwarp();
    uint32_t odd[kChunks] = {};
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
        if (i * 32 >= p.groups) break;
        const int g = i * 32 + lane;
        odd[i] = __ballot_sync(0xffffffffu, g < p.groups && ((first[(g + 1) * p.grp_slabs] - first[g * p.grp_slabs]) >> 1 & 1));
    }
    __syncwarp();
    for (int s = lane; s < slabs; s += 32) {
        // entry s + 1 lies behind s / grp_slabs whole groups, and behind its own where it ends it
        const int g = s / p.grp_slabs, ends = (s + 1) % p.grp_slabs == 0;
        int moved = 0, own = 0;
#pragma unroll
        for (int i = 0; i < kChunks; ++i) {
            const int k = g - i * 32;
            moved += __popc(odd[i] & (k >= 32 ? 0xffffffffu : k > 0 ? (1u << k) - 1 : 0u));
            if ((g >> 5) == i) own = odd[i] >> (g & 31) & ends;
        }
        first[s + 1] += 2 * (moved + own) + own;
    }
}

// One stage of operands into this CTA's ring slot: rows m0.. of A and n0.. of B, k from ks * 128; `bar` is the pair's barrier.
template <int BN>
__device__ __forceinline__ void pair_load_stage(const CUtensorMap* tmA, const CUtensorMap* tmB, uint8_t* a_slot, uint8_t* b_slot,
                                                uint32_t bar, const PairParams& p, int ks, uint32_t live, int m0, int n0, int grp) {
    using namespace pair;
#pragma unroll
    for (int b = 0; b < kPerStage; ++b) {
        if (!(live >> b & 1)) continue;
        const int k0 = (ks * kPerStage + b) * kBK;
        uint8_t* a_dst = a_slot + b * kABytes;
        uint8_t* b_dst = b_slot + b * kBBytes<BN>;
        if (!p.a_mn) {
            tma_load_3d_pair(a_dst, tmA, bar, k0, m0, grp);
        } else {
#pragma unroll
            for (int c = 0; c < 2; ++c) tma_load_3d_pair(a_dst + c * (kBK * 128), tmA, bar, m0 + c * 64, k0, grp);
        }
        if (!p.b_mn) {
            tma_load_3d_pair(b_dst, tmB, bar, k0, n0, grp);
        } else {
#pragma unroll
            for (int c = 0; c < BN / 128; ++c) tma_load_3d_pair(b_dst + c * (kBK * 128), tmB, bar, n0 + c * 64, k0, grp);
        }
    }
}

// What the issuing warp needs to turn a ring slot into MMAs. The whole warp walks the loop, so that descriptors stay in
// uniform registers; one elected lane issues.
template <int BN>
struct PairMma {
    uint64_t a_first, b_first;   // descriptors of the ring's first block
    uint32_t a_step, b_step;     // descriptor distance of 16 k-elements
    uint32_t idesc;
    uint16_t pair_mask;
    bool leader;
    __device__ __forceinline__ PairMma(const PairParams& p, const uint8_t* sA, const uint8_t* sB, uint32_t rank) {
        operands(p, sA, sB);
        pair_mask = static_cast<uint16_t>(3u << rank);
        leader = elect_one();
    }
    // How a product's operands lie in the ring.
    __device__ __forceinline__ void operands(const PairParams& p, const uint8_t* sA, const uint8_t* sB) {
        using namespace pair;
        a_first = umma_smem_desc_sw128(smem_u32(sA), p.a_mn ? kBK * 128 : 0, 1024);
        b_first = umma_smem_desc_sw128(smem_u32(sB), p.b_mn ? kBK * 128 : 0, 1024);
        a_step = (p.a_mn ? kUmmaK * 128 : kUmmaK * 2) >> 4;
        b_step = (p.b_mn ? kUmmaK * 128 : kUmmaK * 2) >> 4;
        idesc = umma_idesc_bf16(kBM, BN, p.a_mn, p.b_mn);
    }
    // The live blocks of slot s into the accumulator; `started` is 0 before the first MMA of a tile, which overwrites it.
    __device__ __forceinline__ void stage(uint32_t d_tmem, int s, uint32_t live, uint32_t& started, uint64_t* empty) {
        using namespace pair;
#pragma unroll
        for (int b = 0; b < kPerStage; ++b) {
            if (!(live >> b & 1)) continue;
            const uint64_t adesc = a_first + static_cast<uint32_t>((s * kPerStage + b) * (kABytes >> 4));
            const uint64_t bdesc = b_first + static_cast<uint32_t>((s * kPerStage + b) * (kBBytes<BN> >> 4));
            if (leader) {
#pragma unroll
                for (int k = 0; k < kBK / kUmmaK; ++k)
                    umma_f16_ss_pair(d_tmem, adesc + k * a_step, bdesc + k * b_step, idesc, k == 0 ? started : 1u);
            }
            started = 1;
        }
        if (leader) umma_commit_pair(empty, pair_mask);
    }
};

// What a kernel's epilogue can do. One kernel with every epilogue and both walks spilled registers and is so long that short products wait for
// its instructions. us, one kernel / one for each kind, plain and ragged: a step of 49 launches 325 / 308, one of 189 launches 4150 / 4000, the expert half of
// a layer on 4068 tokens, 32 experts, 256 x 1152, 148 / 139.
enum PairKind { kPairBf16, kPairF32, kPairSwiglu, kPairAny };   // kPairAny: bf16 and fp32, of two products

template <int BN, int kProducts, PairKind kKind, bool kRagged>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair::kThreads, 1)
gemm_pair_kernel(const __grid_constant__ PairLaunch<kProducts> launch) {
    using namespace pair;
    const PairParams& shared = launch.product[0].p;    // status, overlap and ragged rows are the launch's
    constexpr int STAGES = kStages<BN>;
    constexpr int HALF = BN / 2;          // columns of the tile one epilogue warp drains; rows of B one CTA loads
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + STAGES * kPerStage * kABytes;
    uint8_t* sE = smem + STAGES * kPerStage * kBlock<BN>;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sE + kEpiWarps * kBox);
    uint64_t* full = bars;                      // [STAGES] used in the even CTA: both CTAs' operands of a stage have landed
    uint64_t* empty = bars + STAGES;            // [STAGES] in each CTA: the MMAs that read the stage are done
    uint64_t* tmem_full = bars + 2 * STAGES;    // [2] in each CTA
    uint64_t* tmem_empty = tmem_full + 2;       // [2] used in the even CTA: both CTAs' epilogue warps have read the accumulator
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* first = reinterpret_cast<int*>(sE + kEpiWarps * kBox + 512);   // [slabs + 1] live halves before a slab

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();

    if (warp == 0) {
        // one barrier per lane: in turn they took as long as the TMEM allocation next door
        if (lane < 2 * STAGES + 2) mbar_init(&bars[lane], 1);
        else if (lane < 2 * STAGES + 4) mbar_init(&bars[lane], 2 * kEpiWarps);
        if (lane == 31) *abort_flag = 0;
        mbar_fence_init();
    } else if (warp == 2 && lane == 0) {
#pragma unroll
        for (int i = 0; i < 3 * kProducts; ++i) tma_prefetch_desc(&launch.product[i / 3].map[i % 3]);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 2 * BN);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();      // the other CTA's barriers are initialised before anything arrives on them
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;

    if (kRagged && shared.grp_slabs) {
        if (warp == 3) pair_count_halves(shared, first, lane);
        __syncthreads();
    }
    PairWalk<kProducts, kRagged> tiles(static_cast<int>(blockIdx.x >> 1), static_cast<int>(gridDim.x >> 1));
    int row_half, tn, grp, which; // row_half: first row of this CTA's half of a tile
    bool mine;                   // that half is live

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer (both CTAs)
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            while (ok && tiles.next(launch, first, static_cast<int>(rank), row_half, tn, grp, mine, which)) {
                const PairProduct& product = launch.product[kProducts > 1 ? which : 0];
                const PairParams& p = product.p;
                // SwiGLU: the even CTA brings the gate rows of the weight, the odd one the up rows of the same features
                const int n0 = kKind == kPairSwiglu ? tn * HALF + static_cast<int>(rank) * (p.N >> 1) : tn * BN + static_cast<int>(rank) * HALF;
                PairStages<kRagged> stages(p, grp);
                int ks;
                uint32_t live;
                while (stages.next(p, ks, live)) {
                    if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, shared.status, CAI_DEV_TIMEOUT_TMA_EMPTY)) {
                        ok = false;
                        break;
                    }
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * kBlock<BN> * __popc(live));
                    const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
                    pair_load_stage<BN>(&product.map[0], &product.map[1], sA + s * kPerStage * kABytes, sB + s * kPerStage * kBBytes<BN>, bar, p, ks, live, row_half, n0, grp);
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            if (shared.overlap) grid_dep_launch();
            if (ok) {
                // every stage has been handed back: no arrival of the other CTA is still on its way when this CTA ends
                for (int i = 0; i < STAGES && ok; ++i) {
                    ok = mbar_wait(&empty[s], ph ^ 1, abort_flag, shared.status, CAI_DEV_TIMEOUT_TMA_EMPTY);
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            if (!ok) {
                // Give copies still in flight time to land before the CTA's memory is released.
                for (int i = 0; i < 32; ++i) __nanosleep(50000);
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // ---------------- MMA issuer (even CTA)
            PairMma<BN> mma(shared, sA, sB, 0);
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            int t = 0;
            while (ok && tiles.next(launch, first, static_cast<int>(rank), row_half, tn, grp, mine, which)) {
                const PairParams& p = launch.product[kProducts > 1 ? which : 0].p;
                if (kProducts > 1) mma.operands(p, sA, sB);
                const int acc = t & 1;
                const uint32_t acc_ph = (t >> 1) & 1;
                ++t;
                if (!mbar_wait_warp(&tmem_empty[acc], acc_ph ^ 1, abort_flag, shared.status, CAI_DEV_TIMEOUT_TMEM_EMPTY)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BN;
                uint32_t started = 0;   // 0 for the first MMA of a tile, which overwrites the accumulator
                PairStages<kRagged> stages(p, grp);
                int ks;
                uint32_t live;
                while (stages.next(p, ks, live)) {
                    if (!mbar_wait_warp(&full[s], ph, abort_flag, shared.status, CAI_DEV_TIMEOUT_TMA_FULL)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    mma.stage(d_tmem, s, live, started, &empty[s]);
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok && mma.leader) umma_commit_pair(&tmem_full[acc], mma.pair_mask);
            }
            // both accumulators handed back: no arrival of the odd CTA is still on its way when this one ends
            for (int i = 0; i < 2 && ok; ++i, ++t)
                ok = mbar_wait_warp(&tmem_empty[t & 1], ((t >> 1) & 1) ^ 1, abort_flag, shared.status, CAI_DEV_TIMEOUT_TMEM_EMPTY);
        }
    } else {
        // ---------------- epilogue warps: TMEM -> registers -> shared memory -> TMA
        const int q = warp & 3;              // TMEM lane quarter this warp may read
        const int half = (warp - 2) >> 2;    // which half of the tile's columns
        const int we = warp - 2;
        uint8_t* box = sE + we * kBox;
        const uint32_t box_row = smem_u32(box) + lane * 128;
        const uint32_t sw = static_cast<uint32_t>(lane & 7);
        const uint32_t lane_bits = static_cast<uint32_t>(q * 32) << 16;
        const uint32_t release[2] = {map_to_cta(smem_u32(&tmem_empty[0]), 0), map_to_cta(smem_u32(&tmem_empty[1]), 0)};
        int t = 0;
        bool ok = true;
        while (ok && tiles.next(launch, first, static_cast<int>(rank), row_half, tn, grp, mine, which)) {
            const PairProduct& product = launch.product[kProducts > 1 ? which : 0];
            const PairParams& p = product.p;
            const CUtensorMap &tmC = product.map[2], &tmR = product.map[3];
            const int acc = t & 1;
            const uint32_t acc_ph = (t >> 1) & 1;
            ++t;
            // a weight-gradient tile whose every k-block was skipped has an undefined accumulator: it counts as zero
            bool acc_valid = true;
            if (kRagged && p.seg_mode == 2) {
                PairStages<kRagged> stages(p, grp);
                int ks;
                uint32_t any;
                acc_valid = stages.next(p, ks, any);
            }
            const int row0 = row_half + q * 32;
            const bool live = mine && row0 < p.M;
            const int col_first = tn * BN + half * HALF;
            const bool residual = (kKind == kPairBf16 || kKind == kPairAny) && p.epi == CAI_EPI_BF16_RESIDUAL;
            // the residual of 64 columns, eight lanes to a row of 128 bytes; the first 64 come in while the main loop runs. They reach the lanes that
            // own the rows through the box. (A row per lane met 32 lines a load. us, before / now, without a residual:
            // 3840 x 5456 x 1000 50.6 / 47.9, 43.6; 4096 x 4096 x 1024 32.4 / 31.2, 28.8; 3840 x 1000 x 2728 25.3 / 24.2, 23.3.)
            const __nv_bfloat16* rfirst = p.R + (static_cast<long long>(grp) * p.grp_c + row0 + (lane >> 3)) * p.ldr + (lane & 7) * 8;
            uint4 res[8];
            auto fetch = [&](int col) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (mine && row0 + i * 4 + (lane >> 3) < p.M && col + (lane & 7) * 8 < p.N)
                        res[i] = *reinterpret_cast<const uint4*>(rfirst + static_cast<long long>(i * 4) * p.ldr + col);
            };
            if (residual) fetch(col_first);
            if (!mbar_wait_warp(&tmem_full[acc], acc_ph, abort_flag, shared.status, CAI_DEV_TIMEOUT_TMEM_FULL)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t tacc = tmem_base + lane_bits + acc * BN;
            if (live) {
                if constexpr (kKind == kPairSwiglu) {
                    // columns [0, HALF) are gate, [HALF, BN) up, of features tn * HALF ...; this warp's share is HALF / 2 of each
                    const int F = p.N >> 1;
#pragma unroll 1
                    for (int c = 0; c < HALF / 2; c += 64) {
                        uint32_t g[32], u[32], a[32];
                        const int f0 = half * (HALF / 2) + c, j = tn * HALF + f0;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t rg[32], ru[32];
                            tmem_ld_32x32(tacc + f0 + h * 32, rg);
                            tmem_ld_32x32(tacc + HALF + f0 + h * 32, ru);
                            tmem_ld_wait();
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                // round to bf16 first: the activation is computed from the values the backward will read
                                const uint32_t pg = pack_bf16(__uint_as_float(rg[2 * e]) * p.alpha, __uint_as_float(rg[2 * e + 1]) * p.alpha);
                                const uint32_t pu = pack_bf16(__uint_as_float(ru[2 * e]) * p.alpha, __uint_as_float(ru[2 * e + 1]) * p.alpha);
                                const float g0 = bf16_lo(pg), g1 = bf16_hi(pg), u0 = bf16_lo(pu), u1 = bf16_hi(pu);
                                g[h * 16 + e] = pg;
                                u[h * 16 + e] = pu;
                                a[h * 16 + e] = pack_bf16(g0 * (1.f / (1.f + __expf(-g0))) * u0, g1 * (1.f / (1.f + __expf(-g1))) * u1);
                            }
                        }
                        if (j >= F) continue;
#pragma unroll
                        for (int o = 0; o < 3; ++o) {
                            const uint32_t* v = o == 0 ? g : o == 1 ? u : a;
                            if (lane == 0) tma_store_wait_read0();
                            __syncwarp();
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                st_shared_v4(box_row + ((k ^ sw) << 4), v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (lane == 0) {
                                if (o == 2) tma_store_3d(&tmR, box, j, row0, grp);
                                else tma_store_3d(&tmC, box, j, o, row0);   // gate, up: the halves of a row
                                tma_store_commit();
                            }
                        }
                    }
                } else if (kKind == kPairBf16 || (kKind == kPairAny && (p.epi == CAI_EPI_BF16 || residual))) {
#pragma unroll 1
                    for (int c = 0; c < HALF; c += 64) {
                        const int col = col_first + c;
                        if (col >= p.N) break;
                        uint32_t r[2][32];
                        tmem_ld_32x32(tacc + half * HALF + c, r[0]);
                        tmem_ld_32x32(tacc + half * HALF + c + 32, r[1]);
                        tmem_ld_wait();
                        if (kRagged && !acc_valid) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) r[0][e] = r[1][e] = 0u;
                        }
                        if (lane == 0) tma_store_wait_read0();
                        __syncwarp();
                        if (residual) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const int r4 = i * 4 + (lane >> 3);
                                st_shared_v4(smem_u32(box) + r4 * 128 + (((lane ^ r4) & 7) << 4), res[i].x, res[i].y, res[i].z, res[i].w);
                            }
                            __syncwarp();
                            if (c + 64 < HALF) fetch(col + 64);
                        }
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            float v[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[k >> 2][(k & 3) * 8 + e]) * p.alpha;
                            const uint32_t at = box_row + ((k ^ sw) << 4);
                            if (residual) {
                                const uint4 rv = ld_shared_v4(at);
                                v[0] += bf16_lo(rv.x); v[1] += bf16_hi(rv.x);
                                v[2] += bf16_lo(rv.y); v[3] += bf16_hi(rv.y);
                                v[4] += bf16_lo(rv.z); v[5] += bf16_hi(rv.z);
                                v[6] += bf16_lo(rv.w); v[7] += bf16_hi(rv.w);
                            }
                            st_shared_v4(at, pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_3d(&tmC, box, col, row0, grp);
                            tma_store_commit();
                        }
                    }
                } else {
                    const bool accum = p.epi == CAI_EPI_F32_ACCUM;
#pragma unroll 1
                    for (int c = 0; c < HALF; c += 32) {
                        const int col = col_first + c;
                        if (col >= p.N) break;
                        uint32_t r[32];
                        tmem_ld_32x32(tacc + half * HALF + c, r);
                        tmem_ld_wait();
                        if (lane == 0) tma_store_wait_read0();
                        __syncwarp();
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            uint32_t v[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) v[e] = !kRagged || acc_valid ? __float_as_uint(__uint_as_float(r[4 * k + e]) * p.alpha) : 0u;
                            st_shared_v4(box_row + ((k ^ sw) << 4), v[0], v[1], v[2], v[3]);
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            if (accum) tma_reduce_add_3d(&tmC, box, col, row0, grp);
                            else tma_store_3d(&tmC, box, col, row0, grp);
                            tma_store_commit();
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(release[acc]);
        }
        if (lane == 0) tma_store_wait0();
    }

    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 2 * BN);
    }
}

// ---------------------------------------------------------------------------- split along K
// Few output tiles (short batches, the weight gradients of narrow layers): S pairs, one cluster of 2 S CTAs, share a 256 x 128
// tile, each taking a slice of K. What bounds such a product is how fast one SM can be fed: a CTA of this tile takes in 48 KB
// per 128 k-elements at about 54 B / cycle, twice as long as the MMAs need. The partial accumulators meet in shared memory:
// every CTA leaves its 128 x 128 fp32 partial in its own (the operand ring is free by then), and after a cluster barrier each
// adds up, always in the order of the slices, a 128 / S column slab of all partials of its rows through distributed shared
// memory and writes it. No workspace, no atomics, the same result in every run.
namespace pair {
constexpr int kSplitBN = kSplitCols;
constexpr int kSplitSmem = kStages<kSplitBN> * kPerStage * kBlock<kSplitBN> + 512 + 1024;
}  // namespace pair

// The operands' maps and the rest, of one product or of two. Two products in clusters of 2 S CTAs may be cut into fewer slices than S (each keeps
// the sums of its own form): such a cluster holds S / slices tiles next to each other.
template <int kProducts> struct SplitLaunch {
    CUtensorMap map[kProducts][2];
    PairParams p[kProducts];
    int slices[kProducts];
    int first1;                // the second product's first cluster
};

template <int S, int kProducts>
__global__ void __launch_bounds__(pair::kThreads, 1)
gemm_pair_split_kernel(const __grid_constant__ SplitLaunch<kProducts> launch) {
    using namespace pair;
    int tile = launch.p[0].tile0 + static_cast<int>(blockIdx.x) / (2 * S);   // or, of two products, the cluster's number
    const int which = kProducts > 1 && tile >= launch.first1;
    const PairParams& p = launch.p[which];
    const int slices = kProducts > 1 ? launch.slices[which] : S;
    const CUtensorMap &tmA = launch.map[which][0], &tmB = launch.map[which][1];
    constexpr int BN = kSplitBN, STAGES = kStages<BN>, HALF = BN / 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + STAGES * kPerStage * kABytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * kPerStage * kBlock<BN>);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* tmem_full = bars + 2 * STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t even = rank & ~1u;          // the CTA of my pair that issues
    const int side = static_cast<int>(rank & 1);
    int slice = static_cast<int>(rank >> 1), slice0 = 0;     // my slice of my tile; the pair of the cluster that has its first one
    bool some = true;                                        // this pair has a tile
    if (kProducts > 1) {
        const int mine = slice / slices;
        slice0 = mine * slices;
        slice -= slice0;
        tile = (tile - (which ? launch.first1 : 0)) * (S / slices) + mine;
        some = tile < p.tiles_m * p.tiles_n;
    }

    if (warp == 0) {
        if (lane < 2 * STAGES + 1) mbar_init(&bars[lane], 1);
        if (lane == 31) *abort_flag = 0;
        mbar_fence_init();
    } else if (warp == 2 && lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, BN);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;

    int tm, tn, grp;
    pair_tile_coords(p, tile, tm, tn, grp);
    const int num_kb = (p.K + kBK - 1) / kBK;
    const int num_ks = (num_kb + kPerStage - 1) / kPerStage;
    const int ks0 = some ? num_ks * slice / slices : 0, ks1 = some ? num_ks * (slice + 1) / slices : 0;
    const int row_half = some ? tm * kBM + side * 128 : p.M;

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            const uint32_t full0 = map_to_cta(smem_u32(full), even);
            for (int ks = ks0; ks < ks1; ++ks) {
                const uint32_t live = (ks + 1) * kPerStage <= num_kb ? 3u : 1u;
                if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_EMPTY)) {
                    ok = false;
                    break;
                }
                if (side == 0) mbar_expect_tx(&full[s], 2 * kBlock<BN> * __popc(live));
                pair_load_stage<BN>(&tmA, &tmB, sA + s * kPerStage * kABytes, sB + s * kPerStage * kBBytes<BN>, full0 + s * 8, p, ks, live,
                                    row_half, tn * BN + side * HALF, grp);
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (p.overlap) grid_dep_launch();
            // every stage handed back: no arrival is still on its way when the CTA ends
            for (int i = 0; i < STAGES && ok; ++i) {
                ok = mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_EMPTY);
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (!ok)
                for (int i = 0; i < 32; ++i) __nanosleep(50000);   // let copies in flight land
        }
    } else if (warp == 1) {
        if (side == 0) {
            // ---------------- MMA issuer (even CTA of each pair)
            PairMma<BN> mma(p, sA, sB, even);
            int s = 0;
            uint32_t ph = 0, started = 0;
            bool ok = true;
            for (int ks = ks0; ks < ks1; ++ks) {
                const uint32_t live = (ks + 1) * kPerStage <= num_kb ? 3u : 1u;
                if (!mbar_wait_warp(&full[s], ph, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_FULL)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                mma.stage(tmem_base, s, live, started, &empty[s]);
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (ok && mma.leader) umma_commit_pair(tmem_full, mma.pair_mask);
        }
    } else {
        // ---------------- partial accumulator -> shared memory: row r, 16-byte chunk c at r * 512 + (c ^ (r & 7)) * 16.
        // A CTA without rows waits too: the even CTA's commit arrives on its barrier as well.
        const int q = warp & 3, half = (warp - 2) >> 2;
        const uint32_t dst = smem_u32(smem) + (q * 32 + lane) * (BN * 4);
        const uint32_t tacc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * HALF;
        if (mbar_wait_warp(tmem_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_FULL) && row_half < p.M) {
            tc_fence_after();
            uint32_t r[2][32];
            tmem_ld_32x32(tacc, r[0]);
            tmem_ld_32x32(tacc + 32, r[1]);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < HALF / 4; ++c)
                st_shared_v4(dst + (((half * (HALF / 4) + c) ^ (lane & 7)) << 4), r[c >> 3][(c & 7) * 4], r[c >> 3][(c & 7) * 4 + 1],
                             r[c >> 3][(c & 7) * 4 + 2], r[c >> 3][(c & 7) * 4 + 3]);
        }
    }
    tc_fence_before();
    __syncwarp();
    cluster_sync_memory();     // every partial of the cluster is in place
    if (row_half < p.M && !*abort_flag) {
        const int W = BN / 4 / slices;         // 16-byte chunks of my slab per row
        const int col0 = tn * BN + slice * (BN / slices);
        uint32_t src[S];
#pragma unroll
        for (int i = 0; i < S; ++i) src[i] = map_to_cta(smem_u32(smem), 2 * (i < slices ? slice0 + i : slice0) + side);
#pragma unroll 2
        for (int it = threadIdx.x; it < 128 * W; it += kThreads) {
            const int r = it / W, c = it % W;
            const int row_in = row_half + r, col = col0 + c * 4;
            const uint32_t at = r * (BN * 4) + (((slice * W + c) ^ (r & 7)) << 4);
            if (row_in >= p.M || col >= p.N) continue;   // before the loads: every one issued is consumed before the closing barrier
            float4 part[S];
#pragma unroll
            for (int i = 0; i < S; ++i)
                if (i < slices) part[i] = ld_cluster_f4(src[i] + at);
            float4 v = part[0];
#pragma unroll
            for (int i = 1; i < S; ++i) {
                if (i >= slices) break;
                v.x += part[i].x; v.y += part[i].y; v.z += part[i].z; v.w += part[i].w;
            }
            v.x *= p.alpha; v.y *= p.alpha; v.z *= p.alpha; v.w *= p.alpha;
            const long long row = row_in + static_cast<long long>(grp) * p.grp_c;
            if (p.epi == CAI_EPI_F32 || p.epi == CAI_EPI_F32_ACCUM) {
                float4* dst = reinterpret_cast<float4*>(static_cast<float*>(p.C) + row * p.ldc + col);
                if (p.epi == CAI_EPI_F32_ACCUM) {
                    const float4 old = *dst;
                    v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
                }
                *dst = v;
            } else {
                if (p.epi == CAI_EPI_BF16_RESIDUAL) {
                    const uint2 rv = *reinterpret_cast<const uint2*>(p.R + row * p.ldr + col);
                    v.x += bf16_lo(rv.x); v.y += bf16_hi(rv.x); v.z += bf16_lo(rv.y); v.w += bf16_hi(rv.y);
                }
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
            }
        }
    }
    __syncwarp();
    cluster_sync_memory();     // nobody leaves while another CTA may still read its partial (ordered behind those reads)
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, BN);
    }
}

template <int S>
static void split_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, unsigned grid, bool overlap, cudaStream_t st) {
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(pair::kThreads);
    cfg.dynamicSmemBytes = pair::kSplitSmem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * S;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see launch_early
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 2 : 1;
}

// Tensor map of rows x cols per group, the groups `apart` rows apart.
static bool pair_map(CUtensorMap* m, const GemmShape& g, const void* base, int rows, int cols, long long ld, long long apart, int box_cols,
                     int box_rows, int bytes) {
    return encode_tmap_3d(m, base, cols, rows, g.groups, ld, (g.groups > 1 ? apart : rows) * ld, box_cols, box_rows, bytes);
}
static bool pair_operand_maps(CUtensorMap* tmA, CUtensorMap* tmB, const void* A, const void* B, const GemmShape& g, int bn) {
    const bool ok = !g.a_mn ? pair_map(tmA, g, A, g.M, g.K, g.lda, g.grp_a, 64, 128, 2) : pair_map(tmA, g, A, g.K, g.M, g.lda, g.grp_a, 64, pair::kBK, 2);
    return ok && (!g.b_mn ? pair_map(tmB, g, B, g.N, g.K, g.ldb, g.grp_b, 64, bn / 2, 2)
                          : pair_map(tmB, g, B, g.K, g.N, g.ldb, g.grp_b, 64, pair::kBK, 2));
}

template <typename Kernel>
static bool allow_smem(Kernel kernel, int bytes, const char* what) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess) return true;
    set_last_error("cudaFuncSetAttribute(%s) failed: %s", what, cudaGetErrorString(cudaGetLastError()));
    return false;
}
static int launched(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return CAI_K_OK;
    set_last_error("%s launch failed: %s", what, cudaGetErrorString(e));
    return CAI_K_CUDA;
}
static void pair_tiles(PairParams& p, int tile_cols) {
    p.tiles_m = (p.M + pair::kBM - 1) / pair::kBM;
    p.tiles_n = (p.N + tile_cols - 1) / tile_cols;
    p.group_m = 8;
}

template <int S, int kProducts>
static int launch_split(SplitLaunch<kProducts>& l, int at_once, cudaStream_t st) {
    static bool configured[64] = {};
    const int dev = current_device();
    if (!configured[dev & 63]) {
        if (!allow_smem(gemm_pair_split_kernel<S, kProducts>, pair::kSplitSmem, "gemm_pair_split")) return CAI_K_CUDA;
        configured[dev & 63] = true;
    }
    int tiles = 0;                             // clusters, of two products
    for (int i = 0; i < kProducts; ++i) {
        PairParams& p = l.p[i];
        l.first1 = tiles;
        pair_tiles(p, pair::kSplitBN);
        const int per_cluster = S / l.slices[i];
        tiles += (p.tiles_m * p.tiles_n * p.groups + per_cluster - 1) / per_cluster;
    }
    // Under a limit on the SMs the clusters go out in turns of `at_once`, each launched when the one before has ended: the same sums in the
    // same order.
    for (int& tile0 = l.p[0].tile0; tile0 < tiles; tile0 += at_once) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        split_config<S>(cfg, attr, static_cast<unsigned>(2 * S * (tiles - tile0 < at_once ? tiles - tile0 : at_once)), l.p[0].overlap, st);
        const int rc = launched(cudaLaunchKernelEx(&cfg, gemm_pair_split_kernel<S, kProducts>, l), "gemm_pair_split");
        if (rc) return rc;
    }
    return CAI_K_OK;
}

// What the kernel needs for one product in tiles of BN columns; false if its operands do not fit a tensor map.
template <int BN>
static bool pair_product(PairProduct& q, const void* A, const void* B, const GemmShape& g, const PairParams& p) {
    q.p = p;
    pair_tiles(q.p, BN);
    bool ok = pair_operand_maps(&q.map[0], &q.map[1], A, B, g, BN);
    const bool f32 = p.epi == CAI_EPI_F32 || p.epi == CAI_EPI_F32_ACCUM;
    if (p.epi == CAI_EPI_SWIGLU)
        // a row of C as its gate half and its up half, so that a box of either ends with it: F need not be a multiple of a tile
        return ok && encode_tmap_3d(&q.map[2], g.C, p.N / 2, 2, p.M, p.N / 2, g.ldc, 64, 1, 2, 32) &&
               pair_map(&q.map[3], g, g.R, p.M, p.N / 2, g.ldr, g.grp_c, 64, 32, 2);
    ok = ok && pair_map(&q.map[2], g, g.C, p.M, p.N, g.ldc, g.grp_c, f32 ? 32 : 64, 32, f32 ? 4 : 2);
    q.map[3] = q.map[2];
    return ok;
}

template <int BN, int kProducts, PairKind kKind, bool kRagged>
static int launch_pair(const PairLaunch<kProducts>& l, int pairs, cudaStream_t st) {
    static bool configured[64] = {};
    const int dev = current_device();
    if (!configured[dev & 63]) {
        if (!allow_smem(gemm_pair_kernel<BN, kProducts, kKind, kRagged>, pair::kSmem<BN>, "gemm_pair")) return CAI_K_CUDA;
        configured[dev & 63] = true;
    }
    const int grid = 2 * pairs;
    if (l.product[0].p.overlap) launch_early(gemm_pair_kernel<BN, kProducts, kKind, kRagged>, grid, pair::kThreads, pair::kSmem<BN>, st, l);
    else gemm_pair_kernel<BN, kProducts, kKind, kRagged><<<grid, pair::kThreads, pair::kSmem<BN>, st>>>(l);
    return launched(cudaGetLastError(), "gemm_pair");
}
template <int BN>
static int launch_one(const void* A, const void* B, const GemmShape& g, const PairParams& p, int pairs, cudaStream_t st) {
    PairLaunch<1> l = {};
    if (!pair_product<BN>(l.product[0], A, B, g, p)) return CAI_K_BAD_ARG;
    const int tiles = l.product[0].p.tiles_m * l.product[0].p.tiles_n * p.groups;
    const int at_once = tiles < pairs ? tiles : pairs;
    if constexpr (BN == 256)                        // the only form that has it
        if (p.epi == CAI_EPI_SWIGLU)
            return p.seg_mode ? launch_pair<BN, 1, kPairSwiglu, true>(l, at_once, st) : launch_pair<BN, 1, kPairSwiglu, false>(l, at_once, st);
    if (p.epi == CAI_EPI_F32 || p.epi == CAI_EPI_F32_ACCUM)
        return p.seg_mode ? launch_pair<BN, 1, kPairF32, true>(l, at_once, st) : launch_pair<BN, 1, kPairF32, false>(l, at_once, st);
    return p.seg_mode ? launch_pair<BN, 1, kPairBf16, true>(l, at_once, st) : launch_pair<BN, 1, kPairBf16, false>(l, at_once, st);
}

// Clusters (of 2 CTAs per slice) that one launch may hold: persistent pairs, or tiles of the split form.
static int pair_clusters(const PairForm& f, int sms, int sm_limit) {
    const int cluster = 2 * f.slices;
    if (sm_limit <= 0 && f.slices > 1) return 1 << 20;   // every tile in one launch
    const int n = (sm_limit > 0 && sm_limit < sms ? sm_limit : sms) / cluster;
    return n < 1 ? 1 : n;                                // a cluster is the least that can run
}

// Slabs of a group, where the live halves of all groups' slabs are counted ahead; 0 where they are too many.
static int pair_counted_slabs(int M, int seg_rows, int groups) {
    const long long slabs = (static_cast<long long>(M) + seg_rows - 1) / seg_rows;
    return slabs * groups <= pair::kMaxSlabs ? static_cast<int>(slabs) : 0;
}

static PairParams pair_params(const GemmShape& g, int dev) {
    PairParams p = {};
    p.M = g.M; p.N = g.N; p.K = g.K;
    p.a_mn = g.a_mn; p.b_mn = g.b_mn;
    p.epi = g.epi; p.alpha = g.alpha;
    p.groups = g.groups;
    p.seg_counts = g.seg_counts; p.seg_rows = g.seg_rows; p.seg_mode = g.seg_mode; p.grp_seg = g.grp_seg;
    p.C = g.C;
    p.R = static_cast<const __nv_bfloat16*>(g.R);
    p.ldc = g.ldc; p.ldr = g.ldr; p.grp_c = g.grp_c;
    p.overlap = g.sm_limit <= 0;
    p.grp_slabs = g.seg_mode == 1 ? pair_counted_slabs(g.M, g.seg_rows, g.groups) : 0;
    p.status = status_words(dev);
    return p;
}
template <int S>
static int split_one(const void* A, const void* B, const GemmShape& g, const PairParams& p, int at_once, cudaStream_t st) {
    SplitLaunch<1> l = {};
    l.p[0] = p;
    l.slices[0] = S;
    if (!pair_operand_maps(&l.map[0][0], &l.map[0][1], A, B, g, pair::kSplitBN)) return CAI_K_BAD_ARG;
    return launch_split<S, 1>(l, at_once, st);
}

int gemm_pair(const void* A, const void* B, const GemmShape& g, cudaStream_t st) {
    const int dev = current_device();
    const PairParams p = pair_params(g, dev);
    const PairForm f = pair_form(g.M, g.N, g.K, g.groups, g.epi, g.seg_mode != 0);
    const int at_once = pair_clusters(f, sm_count(dev), g.sm_limit);
    if (f.slices == 4) return split_one<4>(A, B, g, p, at_once, st);
    if (f.slices == 2) return split_one<2>(A, B, g, p, at_once, st);
    return f.tile_cols == 256 ? launch_one<256>(A, B, g, p, at_once, st) : launch_one<128>(A, B, g, p, at_once, st);
}

// Neither may be ragged, of several products or under a limit on the SMs.
bool pair_two_form(const GemmShape& a, const GemmShape& b, PairTwoForm* out) {
    for (const GemmShape* g : {&a, &b})
        if (g->seg_mode || g->groups != 1 || g->sm_limit > 0) return false;
    return pair_two_form(PairShape{a.M, a.N, a.K, a.epi}, PairShape{b.M, b.N, b.K, b.epi}, out);
}

template <int BN>
static int launch_two(const void* const (&A)[2], const void* const (&B)[2], const GemmShape* const (&g)[2], int sms, int dev, cudaStream_t st) {
    PairLaunch<2> l = {};
    long long n[2];
    for (int i = 0; i < 2; ++i) {
        if (!pair_product<BN>(l.product[i], A[i], B[i], *g[i], pair_params(*g[i], dev))) return CAI_K_BAD_ARG;
        n[i] = pair_tile_count(g[i]->M, g[i]->N, BN);
    }
    const long long most = sms / 2 > 0 ? sms / 2 : 1, pairs = n[0] + n[1] < most ? n[0] + n[1] : most;
    pair_two_schedule(n[0], pair_tile_cycles(g[0]->K, BN), n[1], pair_tile_cycles(g[1]->K, BN), pairs, &l.heavier, &l.more_first);
    return launch_pair<BN, 2, kPairAny, false>(l, static_cast<int>(pairs), st);
}
template <int S>
static int split_two(const void* const (&A)[2], const void* const (&B)[2], const GemmShape* const (&g)[2], const int (&slices)[2], int dev, cudaStream_t st) {
    SplitLaunch<2> l = {};
    for (int i = 0; i < 2; ++i) {
        l.p[i] = pair_params(*g[i], dev);
        l.slices[i] = slices[i];
        if (!pair_operand_maps(&l.map[i][0], &l.map[i][1], A[i], B[i], *g[i], pair::kSplitBN)) return CAI_K_BAD_ARG;
    }
    return launch_split<S, 2>(l, 1 << 30, st);
}

int gemm_pair_two(const void* A0, const void* B0, const GemmShape& g0, const void* A1, const void* B1, const GemmShape& g1, const PairTwoForm& f,
                  cudaStream_t st) {
    const int dev = current_device();
    const void *const A[2] = {f.first ? A1 : A0, f.first ? A0 : A1}, *const B[2] = {f.first ? B1 : B0, f.first ? B0 : B1};
    const GemmShape* const g[2] = {f.first ? &g1 : &g0, f.first ? &g0 : &g1};
    const int most = f.slices[0] > f.slices[1] ? f.slices[0] : f.slices[1], slices[2] = {f.slices[f.first], f.slices[1 - f.first]};
    if (most == 4) return split_two<4>(A, B, g, slices, dev, st);
    if (most == 2) return split_two<2>(A, B, g, slices, dev, st);
    return f.tile_cols == 256 ? launch_two<256>(A, B, g, sm_count(dev), dev, st) : launch_two<128>(A, B, g, sm_count(dev), dev, st);
}

}  // namespace cai

using namespace cai;

CAI_API int cai_gemm_bf16_form(int M, int N, int K, int groups, int epi, int segmented, int sms, int sm_limit, int* tile_cols, int* slices,
                               int* ctas) {
    if (M <= 0 || N <= 0 || K <= 0 || groups <= 0 || epi < 0 || epi > CAI_EPI_SWIGLU) return CAI_K_BAD_ARG;
    const PairForm f = pair_form(M, N, K, groups, epi, segmented != 0);
    *tile_cols = f.tile_cols;
    *slices = f.slices;
    const long long tiles = static_cast<long long>((M + pair::kBM - 1) / pair::kBM) * ((N + f.tile_cols - 1) / f.tile_cols) * groups;
    const int at_once = pair_clusters(f, sms, sm_limit);
    *ctas = static_cast<int>(2 * f.slices * (tiles < at_once ? tiles : at_once));
    return CAI_K_OK;
}

CAI_API int cai_gemm_bf16_ragged_walk(int M, int N, int groups, const int* seg_counts, int seg_rows, int tile_cols, int pairs, int pair, int* tiles,
                                      int capacity) {
    if (M <= 0 || N <= 0 || groups <= 0 || !seg_counts || seg_rows <= 0 || seg_rows % 128 || tile_cols <= 0 || pair < 0 || pair >= pairs)
        return CAI_K_BAD_ARG;
    PairParams p = {};
    p.M = M; p.N = N; p.groups = groups;
    p.tiles_m = (M + pair::kBM - 1) / pair::kBM;
    p.tiles_n = (N + tile_cols - 1) / tile_cols;
    p.group_m = 8;
    p.seg_counts = seg_counts; p.seg_rows = seg_rows; p.seg_mode = 1; p.grp_seg = (M + seg_rows - 1) / seg_rows;
    p.grp_slabs = pair_counted_slabs(M, seg_rows, groups);
    int first[pair::kMaxSlabs + 1] = {};
    for (int s = 0, halves = 0, grp0 = 0; s < p.grp_slabs * groups; ++s) {
        halves += pair_live_halves(p, s);
        const bool odd = (s + 1) % p.grp_slabs == 0 && ((halves - grp0) & 1);
        halves += odd;
        first[s + 1] = 2 * halves + odd;
        if ((s + 1) % p.grp_slabs == 0) grp0 = halves;
    }
    PairTiles walk[2] = {PairTiles(pair, pairs), PairTiles(pair, pairs)};
    int n = 0;
    for (;; ++n) {
        int row[2], tn[2], grp[2];
        bool live[2], more[2];
        for (int r = 0; r < 2; ++r) more[r] = walk[r].next(p, first, r, row[r], tn[r], grp[r], live[r]);
        if (more[0] != more[1] || (more[0] && (tn[0] != tn[1] || grp[0] != grp[1]))) return CAI_K_BAD_ARG;   // the CTAs of a pair would part
        if (!more[0]) return n;
        if (n < capacity) {
            int* t = tiles + 6 * n;
            t[0] = grp[0]; t[1] = tn[0]; t[2] = row[0]; t[3] = row[1]; t[4] = live[0]; t[5] = live[1];
        }
    }
}

CAI_API int cai_gemm_bf16_swiglu_pays(int M, int F, int K) { return pair_swiglu_pays(M, F, K); }

CAI_API int cai_gemm_bf16_two_walk(int n0, int k0, int n1, int k1, int tile_cols, int pairs, int pair, int* tiles, int capacity) {
    if (n0 < 0 || n1 < 0 || k0 < k1 || k1 <= 0 || pairs <= 0 || pair < 0 || pair >= pairs) return CAI_K_BAD_ARG;
    int heavier, more_first, n = 0, which, tile;
    pair_two_schedule(n0, pair_tile_cycles(k0, tile_cols), n1, pair_tile_cycles(k1, tile_cols), pairs, &heavier, &more_first);
    for (PairTwoTiles walk(pair, pairs); walk.next(n0, n1, heavier, more_first, which, tile); ++n)
        if (n < capacity) {
            tiles[2 * n] = which;
            tiles[2 * n + 1] = tile;
        }
    return n;
}
