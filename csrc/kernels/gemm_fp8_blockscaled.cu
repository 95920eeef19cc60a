// gemm_fp8_blockscaled.cu - fp8 (e4m3) GEMM with 1x128 / 128x128 block scales on tcgen05.
//
//   C[M,N] = sum over k-blocks kb of  sa[m, kb] * sb[n / 128, kb] * (Aq[m, kb-block] . Bq[n, kb-block])
//
// Aq [M,K] and Bq [N,K] are e4m3, K-major; sa [M, K/128] holds one fp32 scale per row and 128-wide
// k-block (activations), sb [ceil(N/128), K/128] one per 128x128 block (weights). These are not the
// scales the tensor core applies by itself (that format is 32-element UE8M0), so every k-block is
// its own MMA group: the MMA warp issues the four K=32 tcgen05.mma (kind::f8f6f4) of a 128-deep
// block into one of two TMEM buffers, eight epilogue warps read that fp32 partial back with
// tcgen05.ld, scale it and add it to accumulators kept in registers while the tensor core works on
// the next block in the other buffer. TMA (128-byte swizzle, one 128-byte row = 128 k-elements)
// feeds a 4-stage shared-memory ring. Persistent, one CTA per SM, 128x256 tiles; most products run on pairs of CTAs (below).
//
// The reference only names the dtype (`param_dtype fp8e4m3`, include/cai_tensor.h:14-22) and has no
// fp8 arithmetic anywhere.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "cai_kernels.h"
#include "host_common.h"
#include "norm_kernels.cuh"
#include "sm100.cuh"

namespace cai {

namespace f8 {
constexpr int kBM = 128;
constexpr int kBN = 256;
constexpr int kBK = 128;   // e4m3 elements = bytes per row of a stage
constexpr int kUmmaK = 32;
constexpr int kStages = 4;
constexpr int kAStage = kBM * kBK;
constexpr int kBStage = kBN * kBK;
constexpr int kStage = kAStage + kBStage;
constexpr int kThreads = 320;  // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int kSmem = kStages * kStage + 1024 + 256;
}  // namespace f8

struct GemmFp8Params {
    int M, N, K;
    const float* sa;   // [M, K/128]
    const float* sb;   // [ceil(N/128), K/128]
    void* C;
    const void* R;
    long long ldc, ldr;
    int epi;
    int tiles_m, tiles_n;
    int* status;
};

// kind::f8f6f4, A = B = e4m3 (format 0), D = f32, both K-major
__host__ __device__ constexpr uint32_t umma_idesc_e4m3(uint32_t m, uint32_t n) {
    return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void umma_f8_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__global__ void __launch_bounds__(f8::kThreads, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmFp8Params p) {
    using namespace f8;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + kStages * kAStage;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStage);
    uint64_t* full = bars;
    uint64_t* empty = bars + kStages;
    uint64_t* part_full = bars + 2 * kStages;        // [2] a k-block's partial product is in TMEM
    uint64_t* part_empty = bars + 2 * kStages + 2;   // [2] the epilogue warps have read it
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&part_full[a], 1);
            mbar_init(&part_empty[a], 8);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 2 * kBN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const int num_tiles = p.tiles_m * p.tiles_n;
    const int num_kb = p.K / kBK;
    const int cta = blockIdx.x, ncta = gridDim.x;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int tile = cta; tile < num_tiles && ok; tile += ncta) {
                const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_EMPTY)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[s], kStage);
                    tma_load_2d(sA + s * kAStage, &tmA, &full[s], kb * kBK, tm * kBM);
                    tma_load_2d(sB + s * kBStage, &tmB, &full[s], kb * kBK, tn * kBN);
                    if (++s == kStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            grid_dep_launch();
            if (!ok)
                for (int i = 0; i < 32; ++i) __nanosleep(50000);  // let copies in flight land before the CTA's memory goes
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_e4m3(kBM, kBN);
            int s = 0;
            uint32_t ph = 0;
            uint32_t it = 0;  // k-blocks issued by this CTA: TMEM buffer = it & 1
            bool ok = true;
            for (int tile = cta; tile < num_tiles && ok; tile += ncta) {
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const uint32_t buf = it & 1;
                    if (!mbar_wait(&part_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_EMPTY) ||
                        !mbar_wait(&full[s], ph, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_FULL)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_base = smem_u32(sA + s * kAStage), b_base = smem_u32(sB + s * kBStage);
#pragma unroll
                    for (int k = 0; k < kBK / kUmmaK; ++k)
                        umma_f8_ss(tmem_base + buf * kBN, umma_smem_desc_sw128(a_base + k * kUmmaK, 0, 1024),
                                   umma_smem_desc_sw128(b_base + k * kUmmaK, 0, 1024), idesc, k != 0 ? 1u : 0u);
                    umma_commit(&empty[s]);
                    umma_commit(&part_full[buf]);
                    if (++s == kStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else {
        // ---------------- epilogue warps: scale-and-add every k-block, then write the tile
        const int q = warp & 3;           // TMEM lane quarter this warp may read
        const int half = (warp - 2) >> 2; // which 128 columns of the tile
        uint32_t it = 0;
        bool ok = true;
        for (int tile = cta; tile < num_tiles && ok; tile += ncta) {
            const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
            const long long row = static_cast<long long>(tm) * kBM + q * 32 + lane;
            const int col0 = tn * kBN + half * 128;
            const bool row_ok = row < p.M;
            const bool cols_ok = col0 < p.N;
            const float* sa_row = p.sa + (row_ok ? row : 0) * num_kb;
            const float* sb_row = p.sb + static_cast<long long>(cols_ok ? col0 / 128 : 0) * num_kb;
            float acc[128];
#pragma unroll
            for (int e = 0; e < 128; ++e) acc[e] = 0.f;
            float s_next = sa_row[0] * sb_row[0];
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                const uint32_t buf = it & 1;
                const float s = s_next;
                if (kb + 1 < num_kb) s_next = sa_row[kb + 1] * sb_row[kb + 1];
                if (!mbar_wait(&part_full[buf], (it >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_FULL)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * kBN + half * 128;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld_32x32(taddr + c * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[c * 32 + e] = fmaf(s, __uint_as_float(r[e]), acc[c * 32 + e]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&part_empty[buf]);
            }
            if (!ok || !row_ok || !cols_ok) continue;
            if (p.epi == CAI_EPI_F32) {
                float* crow = reinterpret_cast<float*>(p.C) + row * p.ldc + col0;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (col0 + j * 4 >= p.N) break;
                    *reinterpret_cast<float4*>(crow + j * 4) = make_float4(acc[j * 4], acc[j * 4 + 1], acc[j * 4 + 2], acc[j * 4 + 3]);
                }
            } else {
                __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col0;
                const __nv_bfloat16* rrow =
                    p.epi == CAI_EPI_BF16_RESIDUAL ? reinterpret_cast<const __nv_bfloat16*>(p.R) + row * p.ldr + col0 : nullptr;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (col0 + j * 8 >= p.N) break;
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = acc[j * 8 + e];
                    if (rrow) {
                        float rf[8];
                        unpack8(*reinterpret_cast<const uint4*>(rrow + j * 8), rf);
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] += rf[e];
                    }
                    *reinterpret_cast<uint4*>(crow + j * 8) = pack8(v);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 2 * f8::kBN);
}

// ---------------------------------------------------------------------------- pairs of CTAs
// The same product on CTA pairs (a cluster of two, cta_group::2): 256 x 256 tiles, each CTA with 128 rows of A and of B per k-block. What holds the
// one-CTA kernel at 1240 cycles per k-block (512 of MMA) is several things of that size: operands arrive at 54 B / cycle (48 KB: 900 cycles; a CTA
// of a pair takes in 32 KB), shared memory is read and written at 128 B / cycle (768), the one issuing thread spends two waits of 200 to
// 300 cycles per block, and eight epilogue warps read 128 columns each behind four waits. Here two warps issue, one per TMEM buffer, each
// paying its waits under the other's MMAs. What is left is the chain of the epilogue warps (wait, read, add, hand back; a satisfied wait or a read of shared
// memory takes some 200 cycles beside the operand reads) and the round trip to the issuing warps. So: the MMAs of a k-block come in two halves of
// 128 columns with barriers of their own, each read by four warps, 128 columns a thread (eight warps of 232 registers, the launch's 168 and what the
// other warpgroup gives up; sixteen warps of 64 columns had 112; 20 bytes a thread are spilled, 32 with sixteen warps); two reads are in flight per wait; the next part is asked
// for before the last additions, without blocking; scales come in eight k-blocks at a time and are read and multiplied four at a time. Cycles per
// k-block, sixteen warps and whole k-blocks / now: 965 / 820 with two pairs at work, 1100 / 983 with 72. us, bursts of 50: 2000 x 4096 x 14336
// 131 / 118, 9472 x 4096 x 4096 176 / 158 (one CTA per tile 145 for the former); with results that leave by TMA through boxes of shared memory,
// for which the ring gave up its sixth stage, instead of 32 lines a store 116 / 150 (a tile's end 8.8 -> 6.5 us). Tried on top: a half per issuing warp (911 and 1075 cycles: four
// waits per k-block instead of three), scales two at a time (872 and 1028), halves with sixteen warps (no change), additions in pairs
// (fma.rn.f32x2; sixteen warps, 131 -> 145 us).
namespace f8p {
constexpr int kBM = 256, kBN = 256, kBK = 128;
constexpr int kStages = 5;
constexpr int kHalf = 128 * kBK;                   // bytes of A, or of B, a CTA brings in per stage
constexpr int kEpiWarps = 8;
constexpr int kThreads = 128 + kEpiWarps * 32;     // warp 0 TMA, warps 1-2 MMA, warp 3 scales, warps 4-11 epilogue
constexpr int kScaleKb = 8;                        // k-blocks whose scales come in at a time
constexpr int kScaleRow = 12;                      // a row of A's eight scales, padded: eight rows' 16 bytes fall on 32 banks
constexpr int kScaleWords = 128 * kScaleRow + 2 * kScaleKb;
constexpr int kBox = 4096;                         // a warp's box of results: 32 rows x 128 bytes
constexpr int kSmem = kStages * 2 * kHalf + kEpiWarps * kBox + 2 * kScaleWords * 4 + 512 + 1024;
}  // namespace f8p

__device__ __forceinline__ void umma_f8_ss_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m, uint32_t cluster_bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2"
        " [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(m), "r"(cluster_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(f8p::kThreads, 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                     const GemmFp8Params p) {
    using namespace f8p;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + kStages * kHalf;
    uint8_t* sE = smem + kStages * 2 * kHalf;
    float* scales = reinterpret_cast<float*>(sE + kEpiWarps * kBox);        // [2][kScaleWords]
    uint64_t* bars = reinterpret_cast<uint64_t*>(scales + 2 * kScaleWords);
    uint64_t* full = bars;                         // [kStages] used in the even CTA: both CTAs' operands have landed
    uint64_t* empty = bars + kStages;              // [kStages] in each CTA
    uint64_t* sc_full = bars + 2 * kStages;        // [2] in each CTA
    uint64_t* part_full = sc_full + 2;             // [buffer][half] in each CTA: that half of a k-block's partial product is in TMEM
    uint64_t* part_empty = part_full + 4;          // [buffer][half] used in the even CTA: both CTAs' epilogue warps have read it
    uint64_t* sc_empty = part_empty + 4;           // [2] in each CTA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    if (warp == 0) {
        constexpr int kParts = 2 * kStages + 6;    // full, empty, scales and parts that arrive
        if (lane < kParts) mbar_init(&bars[lane], 1);
        else if (lane < kParts + 4) mbar_init(&bars[lane], kEpiWarps);         // half of the warps of either CTA
        else if (lane < kParts + 6) mbar_init(&bars[lane], kEpiWarps);
        if (lane == 31) *abort_flag = 0;
        mbar_fence_init();
    } else if (warp == 2 && lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        tma_prefetch_desc(&tmC);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 2 * kBN);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();      // the other CTA's barriers are initialised before anything arrives on them
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const int num_tiles = p.tiles_m * p.tiles_n;
    const int num_kb = p.K / kBK;
    const int first = static_cast<int>(blockIdx.x >> 1), stride = static_cast<int>(gridDim.x >> 1);
    // eight row tiles share a column of B before the next one
    auto coords = [&](int tile, int& tm, int& tn) {
        const int per_group = 8 * p.tiles_n, g = tile / per_group, in = tile - g * per_group;
        const int gsz = min(p.tiles_m - g * 8, 8);
        tm = g * 8 + in % gsz;
        tn = in / gsz;
    };

    if (warp < 4) {
        // 40 + 2 x 232 registers a thread of each of the three warpgroups: the 3 x 168 of the launch
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0) {
            if (lane == 0) {
                // ---------------- TMA producer (both CTAs)
                int s = 0;
                uint32_t ph = 0;
                bool ok = true;
                for (int tile = first; tile < num_tiles && ok; tile += stride) {
                    int tm, tn;
                    coords(tile, tm, tn);
                    const int m0 = tm * kBM + static_cast<int>(rank) * 128, n0 = tn * kBN + static_cast<int>(rank) * 128;
                    for (int kb = 0; kb < num_kb; ++kb) {
                        if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_EMPTY)) {
                            ok = false;
                            break;
                        }
                        if (rank == 0) mbar_expect_tx(&full[s], 4 * kHalf);
                        const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
                        tma_load_2d_pair(sA + s * kHalf, &tmA, bar, kb * kBK, m0);
                        tma_load_2d_pair(sB + s * kHalf, &tmB, bar, kb * kBK, n0);
                        if (++s == kStages) {
                            s = 0;
                            ph ^= 1;
                        }
                    }
                }
                grid_dep_launch();
                // every stage handed back: no arrival of the other CTA is still on its way when this CTA ends
                for (int i = 0; i < kStages && ok; ++i) {
                    ok = mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_EMPTY);
                    if (++s == kStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (!ok)
                    for (int i = 0; i < 32; ++i) __nanosleep(50000);   // let copies in flight land
            }
        } else if (warp < 3) {
            if (rank == 0) {
                // ---------------- MMA issuers (even CTA): warp 1 the even k-blocks into TMEM buffer 0, warp 2 the odd ones into buffer 1
                const uint32_t buf = warp - 1;
                const uint32_t idesc = umma_idesc_e4m3(kBM, kBN / 2);
                const uint64_t a_first = umma_smem_desc_sw128(smem_u32(sA), 0, 1024), b_first = umma_smem_desc_sw128(smem_u32(sB), 0, 1024);
                const bool leader = elect_one();
                const uint32_t total = static_cast<uint32_t>(num_kb) * static_cast<uint32_t>(first < num_tiles ? (num_tiles - first + stride - 1) / stride : 0);
                uint32_t s = buf, ph = 0, n = 0;      // ring slot and its phase; k-blocks this warp has issued
                bool ok = true;
                for (uint32_t it = buf; it < total && ok; it += 2, ++n) {
                    if (!mbar_wait_warp(&full[s], ph, abort_flag, p.status, CAI_DEV_TIMEOUT_TMA_FULL)) {
                        ok = false;
                        break;
                    }
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const uint32_t part = buf * 2 + half;
                        if (!mbar_wait_warp(&part_empty[part], (n & 1) ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_EMPTY)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        if (leader) {
                            const uint64_t ad = a_first + s * (kHalf >> 4), bd = b_first + s * (kHalf >> 4) + half * (kHalf >> 5);
#pragma unroll
                            for (int k = 0; k < kBK / f8::kUmmaK; ++k)
                                umma_f8_ss_pair(tmem_base + part * (kBN / 2), ad + k * (f8::kUmmaK >> 4), bd + k * (f8::kUmmaK >> 4), idesc, k != 0 ? 1u : 0u);
                            umma_commit_pair(&part_full[part], 3);
                            if (half) umma_commit_pair(&empty[s], 3);
                        }
                    }
                    s += 2;
                    if (s >= kStages) {
                        s -= kStages;
                        ph ^= 1;
                    }
                }
                // both parts handed back: no arrival of the odd CTA is still on its way when this one ends
                for (int half = 0; half < 2 && ok; ++half)
                    ok = mbar_wait_warp(&part_empty[buf * 2 + half], (n & 1) ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_EMPTY);
            }
        } else {
            // ---------------- scales of eight k-blocks at a time: lane l takes k-block l & 7 of rows l / 8, l / 8 + 4, ...
            uint32_t b = 0, ph = 0;
            bool ok = true;
            for (int tile = first; tile < num_tiles && ok; tile += stride) {
                int tm, tn;
                coords(tile, tm, tn);
                const int r0 = tm * kBM + static_cast<int>(rank) * 128 + (lane >> 3);
                for (int kb0 = 0; kb0 < num_kb; kb0 += kScaleKb) {
                    if (!mbar_wait_warp(&sc_empty[b], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_EMPTY)) {
                        ok = false;
                        break;
                    }
                    float* dst = scales + b * kScaleWords;
                    const int kb = kb0 + (lane & 7);
                    if (kb < num_kb) {
#pragma unroll 8
                        for (int i = 0; i < 32; ++i)
                            cp_async4(dst + ((lane >> 3) + 4 * i) * kScaleRow + (lane & 7),
                                      p.sa + static_cast<long long>(min(r0 + 4 * i, p.M - 1)) * num_kb + kb);
                        if (lane < 16) {
                            const int cb = min(tn * 2 + (lane >> 3), (p.N - 1) / 128);
                            cp_async4(dst + 128 * kScaleRow + lane, p.sb + static_cast<long long>(cb) * num_kb + kb);
                        }
                    }
                    cp_async_wait_all();
                    mbar_arrive_warp(&sc_full[b]);
                    b ^= 1;
                    if (b == 0) ph ^= 1;
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        // ---------------- epilogue warps: scale-and-add every k-block, then write the tile; 128 columns each.
        // The MMA of a half takes 64 rows of B from either CTA: its 128 columns are 64 of the tile's first 128 and 64 of its second.
        const int q = warp & 3, half = (warp - 4) >> 2;
        const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * (kBN / 2);
        const uint32_t release0 = map_to_cta(smem_u32(&part_empty[half]), 0);
        uint8_t* box = sE + (warp - 4) * kBox;
        const uint32_t box_row = smem_u32(box) + lane * 128, sw = lane & 7;
        uint32_t it = 0, sb = 0, sph = 0;
        bool ok = true, ready = false;     // ready: the next part was seen in tensor memory
        for (int tile = first; tile < num_tiles && ok; tile += stride) {
            float acc[128];
#pragma unroll
            for (int e = 0; e < 128; ++e) acc[e] = 0.f;
            for (int kb0 = 0; kb0 < num_kb && ok; kb0 += 4) {
                const int at = kb0 & (kScaleKb - 1);
                if (at == 0 && !mbar_wait_warp(&sc_full[sb], sph, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_FULL)) {
                    ok = false;
                    break;
                }
                float s0[4], s1[4];
                {
                    const float* sc = scales + sb * kScaleWords;
                    const float4 a = *reinterpret_cast<const float4*>(sc + (q * 32 + lane) * kScaleRow + at);
                    const float4 b0 = *reinterpret_cast<const float4*>(sc + 128 * kScaleRow + at);
                    const float4 b1 = *reinterpret_cast<const float4*>(sc + 128 * kScaleRow + kScaleKb + at);
                    s0[0] = a.x * b0.x; s0[1] = a.y * b0.y; s0[2] = a.z * b0.z; s0[3] = a.w * b0.w;
                    s1[0] = a.x * b1.x; s1[1] = a.y * b1.y; s1[2] = a.z * b1.z; s1[3] = a.w * b1.w;
                }
                if (at || kb0 + 4 >= num_kb) {
                    mbar_arrive_warp(&sc_empty[sb]);
                    sb ^= 1;
                    if (sb == 0) sph ^= 1;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i, ++it) {
                    if (kb0 + i >= num_kb) break;
                    const uint32_t buf = it & 1;
                    if (!ready && !mbar_wait_warp(&part_full[buf * 2 + half], (it >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_TMEM_FULL)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    uint32_t r0[32], r1[32];
                    const uint32_t ta = taddr0 + buf * kBN;
                    tmem_ld_32x32(ta, r0);
                    tmem_ld_32x32(ta + 32, r1);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[e] = fmaf(s0[i], __uint_as_float(r0[e]), acc[e]);
                    tmem_ld_32x32(ta + 64, r0);
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[32 + e] = fmaf(s0[i], __uint_as_float(r1[e]), acc[32 + e]);
                    tmem_ld_32x32(ta + 96, r1);
                    tmem_ld_wait();
                    // read: the buffer goes back before the last additions, and the next part is asked for under them
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(release0 + buf * 16);
                    const bool next = mbar_test_wait(&part_full[(buf ^ 1) * 2 + half], ((it + 1) >> 1) & 1);
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[64 + e] = fmaf(s1[i], __uint_as_float(r0[e]), acc[64 + e]);
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[96 + e] = fmaf(s1[i], __uint_as_float(r1[e]), acc[96 + e]);
                    ready = __all_sync(0xffffffffu, next);
                }
            }
            if (!ok) break;
            int tm, tn;
            coords(tile, tm, tn);
            // through a box of shared memory by TMA, edges clipped by the tensor map: whole lines, and the registers are free for the next tile
            // as soon as the last box is written
            const int row0 = tm * kBM + static_cast<int>(rank) * 128 + q * 32;
            if (row0 >= p.M) continue;
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int col0 = tn * kBN + side * 128 + half * 64;
                if (col0 >= p.N) break;
                if (p.epi == CAI_EPI_F32) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (col0 + h * 32 >= p.N) break;
                        if (lane == 0) tma_store_wait_read0();
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float* v = acc + side * 64 + h * 32 + j * 4;
                            st_shared_v4(box_row + ((j ^ sw) << 4), __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tmC, box, col0 + h * 32, row0);
                            tma_store_commit();
                        }
                    }
                } else {
                    const __nv_bfloat16* rrow = p.epi == CAI_EPI_BF16_RESIDUAL && row0 + lane < p.M
                                                    ? reinterpret_cast<const __nv_bfloat16*>(p.R) + static_cast<long long>(row0 + lane) * p.ldr + col0
                                                    : nullptr;
                    if (lane == 0) tma_store_wait_read0();
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float v[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = acc[side * 64 + j * 8 + e];
                        if (rrow && col0 + j * 8 < p.N) {
                            float rf[8];
                            unpack8(*reinterpret_cast<const uint4*>(rrow + j * 8), rf);
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] += rf[e];
                        }
                        const uint4 o = pack8(v);
                        st_shared_v4(box_row + ((j ^ sw) << 4), o.x, o.y, o.z, o.w);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(&tmC, box, col0, row0);
                        tma_store_commit();
                    }
                }
            }
        }
        if (lane == 0) tma_store_wait0();
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 2 * kBN);
    }
}

// ------------------------------------------------------------------ quantisation
// One warp per (row, 128-column block): amax -> scale = amax / 448, q = x / scale.
__global__ void __launch_bounds__(256)
quant_rows_1x128_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, __nv_fp8_storage_t* __restrict__ q, long long ldq,
                        float* __restrict__ scale, int rows, int cols) {
    grid_dep_begin();
    const int kb_n = cols / 128;
    const long long w = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= static_cast<long long>(rows) * kb_n) return;
    const long long r = w / kb_n;
    const int kb = static_cast<int>(w % kb_n);
    const uint2 raw = *reinterpret_cast<const uint2*>(x + r * ldx + kb * 128 + lane * 4);
    float v[4] = {bf16_lo(raw.x), bf16_hi(raw.x), bf16_lo(raw.y), bf16_hi(raw.y)};
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    amax = warp_max(amax);
    const float s = amax > 0.f ? amax / 448.f : 1.f;
    const float inv = 1.f / s;
    uint32_t out = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e)
        out |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(v[e] * inv, __NV_SATFINITE, __NV_E4M3)) << (8 * e);
    *reinterpret_cast<uint32_t*>(q + r * ldq + kb * 128 + lane * 4) = out;
    if (lane == 0) scale[r * kb_n + kb] = s;
}

__device__ __forceinline__ uint32_t abs_bf16x2(uint32_t v) { return v & 0x7FFF7FFFu; }
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&m);
}
// Largest magnitude (as two bf16, the larger one counts) of eight.
__device__ __forceinline__ uint32_t amax8(const uint4& v) {
    return max_bf16x2(max_bf16x2(abs_bf16x2(v.x), abs_bf16x2(v.y)), max_bf16x2(abs_bf16x2(v.z), abs_bf16x2(v.w)));
}
__device__ __forceinline__ float amax_of(uint32_t m) { return fmaxf(bf16_lo(m), bf16_hi(m)); }
// Eight bf16 times inv as e4m3.
__device__ __forceinline__ uint2 quant8(const uint4& v, float inv) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        h[k] = __nv_cvt_float2_to_fp8x2(make_float2(bf16_lo(w[k]) * inv, bf16_hi(w[k]) * inv), __NV_SATFINITE, __NV_E4M3);
    return make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
}

// The same by 16 lanes per 128-column block, 16 bytes a lane, four blocks in flight per thread. What bounds this is bytes in
// flight (the kernel above has 256 per warp, behind a division of 64-bit numbers). Measured, 8192 x 14336: 144 -> 62 us (2.4
// -> 5.6 TB/s), 2000 x 14336: 36 -> 20 us. Rows of 16-byte aligned pieces only; the kernel above takes the rest.
constexpr int kQuantUnroll = 4;
__global__ void __launch_bounds__(256)
quant_rows_vec_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, __nv_fp8_storage_t* __restrict__ q, long long ldq,
                      float* __restrict__ scale, unsigned blocks, unsigned kb_n) {
    grid_dep_begin();
    const int sub = threadIdx.x & 15;
    // half-warps of a CTA take consecutive blocks, kQuantUnroll times over
    const unsigned b0 = blockIdx.x * (16u * kQuantUnroll) + (threadIdx.x >> 4);
    uint4 v[kQuantUnroll];
    long long row[kQuantUnroll];
    unsigned col[kQuantUnroll];
#pragma unroll
    for (int i = 0; i < kQuantUnroll; ++i) {
        const unsigned b = b0 + 16u * i, r = b / kb_n;
        row[i] = r;
        col[i] = (b - r * kb_n) * 128u + sub * 8;
        v[i] = make_uint4(0, 0, 0, 0);
        if (b < blocks) v[i] = *reinterpret_cast<const uint4*>(x + row[i] * ldx + col[i]);
    }
#pragma unroll
    for (int i = 0; i < kQuantUnroll; ++i) {
        const unsigned b = b0 + 16u * i;
        uint32_t m = amax8(v[i]);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) m = max_bf16x2(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float amax = amax_of(m);
        const float s = amax > 0.f ? amax / 448.f : 1.f;
        if (b < blocks) {
            *reinterpret_cast<uint2*>(q + row[i] * ldq + col[i]) = quant8(v[i], 1.f / s);
            if (sub == 0) scale[b] = s;
        }
    }
}

// One CTA per 128x128 block of a weight [rows, cols]: a common scale; optionally also writes the
// transposed quantised block (qt [cols, rows], for the input-gradient GEMM that contracts over rows).
__global__ void __launch_bounds__(256)
quant_blocks_128x128_kernel(const __nv_bfloat16* __restrict__ w, long long ldw, __nv_fp8_storage_t* __restrict__ q, long long ldq,
                            __nv_fp8_storage_t* __restrict__ qt, long long ldqt, float* __restrict__ scale,
                            float* __restrict__ scale_t, int rows, int cols) {
    grid_dep_begin();
    __shared__ __nv_bfloat16 tile[128][130];
    __shared__ float red[8];
    const int bc = blockIdx.x, br = blockIdx.y;
    const int nbc = gridDim.x, nbr = gridDim.y;
    float amax = 0.f;
    for (int i = threadIdx.x; i < 128 * 128; i += 256) {
        const int r = i >> 7, c = i & 127;
        const long long gr = static_cast<long long>(br) * 128 + r;
        const int gc = bc * 128 + c;
        const float v = (gr < rows && gc < cols) ? __bfloat162float(w[gr * ldw + gc]) : 0.f;
        tile[r][c] = __float2bfloat16(v);
        amax = fmaxf(amax, fabsf(v));
    }
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = red[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) amax = fmaxf(amax, red[k]);
    const float s = amax > 0.f ? amax / 448.f : 1.f;
    const float inv = 1.f / s;
    if (threadIdx.x == 0) {
        scale[static_cast<long long>(br) * nbc + bc] = s;
        if (scale_t) scale_t[static_cast<long long>(bc) * nbr + br] = s;
    }
    for (int i = threadIdx.x; i < 128 * 128; i += 256) {
        const int r = i >> 7, c = i & 127;
        const long long gr = static_cast<long long>(br) * 128 + r;
        const int gc = bc * 128 + c;
        if (gr < rows && gc < cols) q[gr * ldq + gc] = __nv_cvt_float_to_fp8(__bfloat162float(tile[r][c]) * inv, __NV_SATFINITE, __NV_E4M3);
    }
    if (qt)
        for (int i = threadIdx.x; i < 128 * 128; i += 256) {
            const int c = i >> 7, r = i & 127;   // consecutive threads walk a column of the block = a row of qt
            const long long gr = static_cast<long long>(br) * 128 + r;
            const int gc = bc * 128 + c;
            if (gr < rows && gc < cols)
                qt[static_cast<long long>(gc) * ldqt + gr] = __nv_cvt_float_to_fp8(__bfloat162float(tile[r][c]) * inv, __NV_SATFINITE, __NV_E4M3);
        }
}

// The same with 16-byte loads kept in registers, 8-byte stores, and the transposed block turned in shared memory: a thread
// reads a 16 x 4 patch of bytes, transposes it by byte permutations and writes 16 bytes to each of four rows of qt, eight
// lanes filling a 128-byte line. One byte per store bound the kernel above. Word w of row r sits at w ^ (r / 16 * 4), which
// keeps both sides free of bank conflicts. Measured with the transposed copy: 28672 x 4096 373 -> 76 us (1.3 -> 6.2 TB/s),
// 4096 x 14336 203 -> 41 us. Needs cols % 8 == 0 and, for the transposed block, rows % 16 == 0, with the leading dimensions and
// pointers to match; the kernel above takes the rest.
__global__ void __launch_bounds__(256)
quant_blocks_vec_kernel(const __nv_bfloat16* __restrict__ w, long long ldw, __nv_fp8_storage_t* __restrict__ q, long long ldq,
                        __nv_fp8_storage_t* __restrict__ qt, long long ldqt, float* __restrict__ scale,
                        float* __restrict__ scale_t, int rows, int cols) {
    grid_dep_begin();
    __shared__ __align__(16) uint32_t tile[128 * 32];
    __shared__ float red[8];
    const int bc = blockIdx.x, br = blockIdx.y;
    const int nbc = gridDim.x, nbr = gridDim.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r_in = threadIdx.x >> 4, c8 = threadIdx.x & 15;   // rows r_in + 16 i, columns c8 * 8 ...
    const int gc = bc * 128 + c8 * 8;
    uint4 v[8];
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const long long gr = static_cast<long long>(br) * 128 + r_in + 16 * i;
        v[i] = make_uint4(0, 0, 0, 0);
        if (gr < rows && gc < cols) v[i] = *reinterpret_cast<const uint4*>(w + gr * ldw + gc);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) m = max_bf16x2(m, amax8(v[i]));
    float amax = warp_max(amax_of(m));
    if (lane == 0) red[warp] = amax;
    __syncthreads();
    amax = red[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) amax = fmaxf(amax, red[k]);
    const float s = amax > 0.f ? amax / 448.f : 1.f;
    const float inv = 1.f / s;
    if (threadIdx.x == 0) {
        scale[static_cast<long long>(br) * nbc + bc] = s;
        if (scale_t) scale_t[static_cast<long long>(bc) * nbr + br] = s;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = r_in + 16 * i;
        const long long gr = static_cast<long long>(br) * 128 + r;
        const uint2 o = quant8(v[i], inv);
        if (gr < rows && gc < cols) *reinterpret_cast<uint2*>(q + gr * ldq + gc) = o;
        if (qt) *reinterpret_cast<uint2*>(&tile[r * 32 + ((c8 * 2) ^ (i * 4))]) = o;   // r / 16 == i
    }
    if (!qt) return;
    __syncthreads();
    const int rg = lane & 7, cw = warp * 4 + (lane >> 3);   // rows rg * 16 ..., columns cw * 4 ...
    uint32_t out[4][4];                                     // [column][four rows each]
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint32_t a[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) a[t] = tile[(rg * 16 + k * 4 + t) * 32 + (cw ^ (rg * 4))];
        const uint32_t lo01 = __byte_perm(a[0], a[1], 0x5140), hi01 = __byte_perm(a[0], a[1], 0x7362);
        const uint32_t lo23 = __byte_perm(a[2], a[3], 0x5140), hi23 = __byte_perm(a[2], a[3], 0x7362);
        out[0][k] = __byte_perm(lo01, lo23, 0x5410);
        out[1][k] = __byte_perm(lo01, lo23, 0x7632);
        out[2][k] = __byte_perm(hi01, hi23, 0x5410);
        out[3][k] = __byte_perm(hi01, hi23, 0x7632);
    }
    const long long gr = static_cast<long long>(br) * 128 + rg * 16;
    if (gr >= rows) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = bc * 128 + cw * 4 + j;
        if (c < cols)
            *reinterpret_cast<uint4*>(qt + static_cast<long long>(c) * ldqt + gr) = make_uint4(out[j][0], out[j][1], out[j][2], out[j][3]);
    }
}

static bool aligned_to(const void* p, uintptr_t n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }

}  // namespace cai

using namespace cai;

CAI_API int cai_gemm_fp8_blockscaled(const void* Aq, const float* sa, const void* Bq, const float* sb, void* C, const void* R,
                                     int M, int N, int K, long long lda, long long ldb, long long ldc, long long ldr, int epi,
                                     void* stream) {
    if (M <= 0 || N <= 0 || K <= 0) return CAI_K_OK;
    if ((K % 128) || (lda & 15) || (ldb & 15) || (N & 7) || (epi != CAI_EPI_BF16 && epi != CAI_EPI_F32 && epi != CAI_EPI_BF16_RESIDUAL) ||
        (epi != CAI_EPI_F32 && (ldc & 7)) || (epi == CAI_EPI_F32 && (ldc & 3)) || (epi == CAI_EPI_BF16_RESIDUAL && (!R || (ldr & 7)))) {
        set_last_error("gemm_fp8: K %% 128, lda/ldb %% 16, N %% 8 and an aligned C are required (M=%d N=%d K=%d)", M, N, K);
        return CAI_K_BAD_ARG;
    }
    const int dev = current_device();
    const int sms = sm_count(dev);
    // Pairs of CTAs, unless the last half of their 256-row tiles stays empty and costs waves: a wave of pair tiles takes some eight tenths
    // of one of one-CTA tiles of half the rows (us, one-CTA / pair: 2000 x 4096 x 14336 145 / 116, 128 x 14336 x 4096 27.4 / 25.3, 16 x 4096
    // x 4096 22.9 / 19.9; two waves of pairs against one: 128 x 28672 x 4096 31.7 / 47.8). Both forms give the same bits.
    const long long cols = (N + f8::kBN - 1) / f8::kBN, pairs = sms / 2 > 0 ? sms / 2 : 1;
    const long long waves_one = ((M + f8::kBM - 1) / f8::kBM * cols + sms - 1) / sms, waves_pair = ((M + f8p::kBM - 1) / f8p::kBM * cols + pairs - 1) / pairs;
    const bool pair = 8 * waves_pair <= 10 * waves_one;
    CUtensorMap tmA, tmB, tmC;
    const int c_bytes = epi == CAI_EPI_F32 ? 4 : 2;
    if ((pair && !encode_tmap_2d(&tmC, C, M, N, ldc, 128 / c_bytes, 32, c_bytes)) || !encode_tmap_2d(&tmA, Aq, M, K, lda, f8::kBK, 128, 1) || !encode_tmap_2d(&tmB, Bq, N, K, ldb, f8::kBK, pair ? 128 : f8::kBN, 1))
        return CAI_K_BAD_ARG;
    static bool configured[64] = {};
    if (!configured[dev & 63]) {
        if (cudaFuncSetAttribute(gemm_fp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, f8::kSmem) != cudaSuccess ||
            cudaFuncSetAttribute(gemm_fp8_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, f8p::kSmem) != cudaSuccess) {
            set_last_error("cudaFuncSetAttribute(gemm_fp8) failed");
            return CAI_K_CUDA;
        }
        configured[dev & 63] = true;
    }
    GemmFp8Params p;
    p.M = M; p.N = N; p.K = K;
    p.sa = sa; p.sb = sb;
    p.C = C; p.R = R; p.ldc = ldc; p.ldr = ldr; p.epi = epi;
    const int rows = pair ? f8p::kBM : f8::kBM;
    p.tiles_m = (M + rows - 1) / rows;
    p.tiles_n = static_cast<int>(cols);
    p.status = status_words(dev);
    const int tiles = p.tiles_m * p.tiles_n;
    if (pair) {
        launch_early(gemm_fp8_pair_kernel, 2 * (tiles < pairs ? tiles : static_cast<int>(pairs)), f8p::kThreads, f8p::kSmem,
                     static_cast<cudaStream_t>(stream), tmA, tmB, tmC, p);
    } else {
        launch_early(gemm_fp8_kernel, tiles < sms ? tiles : sms, f8::kThreads, f8::kSmem, static_cast<cudaStream_t>(stream), tmA, tmB, p);
    }
    if (cudaGetLastError() != cudaSuccess) {
        set_last_error("gemm_fp8 launch failed");
        return CAI_K_CUDA;
    }
    return CAI_K_OK;
}

CAI_API int cai_quant_rows_1x128(const void* x, long long ldx, void* q, long long ldq, float* scale, int rows, int cols,
                                 void* stream) {
    if (cols % 128 || (ldx & 3) || (ldq & 3)) {
        set_last_error("quant_rows: columns must be a multiple of 128");
        return CAI_K_BAD_ARG;
    }
    const long long warps = static_cast<long long>(rows) * (cols / 128);
    if (warps == 0) return CAI_K_OK;
    if (warps < (1ll << 31) && !(ldx & 7) && !(ldq & 7) && aligned_to(x, 16) && aligned_to(q, 8)) {
        constexpr unsigned per_cta = 16u * kQuantUnroll;
        // Launched the ordinary way: early, behind a GEMM on CTA pairs and in front of the product above, it gains nothing (the three, four times
        // over, in ms, ordinary / early: 8192 x 4096 x 28672 9.6-10.0 / 9.9-10.3, 8192 x 28672 x 4096 5.3-5.6 / 5.6, 2048 x 4096 x 14336 1.36 /
        // 1.36). While that product ran on one CTA a tile throughout, it took half as long again behind an early quantiser.
        quant_rows_vec_kernel<<<static_cast<unsigned>((warps + per_cta - 1) / per_cta), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_fp8_storage_t*>(q), ldq, scale, static_cast<unsigned>(warps),
            static_cast<unsigned>(cols / 128));
        return cudaGetLastError() == cudaSuccess ? 0 : CAI_K_CUDA;
    }
    quant_rows_1x128_kernel<<<static_cast<unsigned>((warps * 32 + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_fp8_storage_t*>(q), ldq, scale, rows, cols);
    return cudaGetLastError() == cudaSuccess ? 0 : CAI_K_CUDA;
}

CAI_API int cai_quant_blocks_128x128(const void* w, long long ldw, void* q, long long ldq, void* qt, long long ldqt, float* scale,
                                     float* scale_t, int rows, int cols, void* stream) {
    if (rows <= 0 || cols <= 0) return CAI_K_OK;
    dim3 grid((cols + 127) / 128, (rows + 127) / 128);
    if (!(cols & 7) && !(ldw & 7) && !(ldq & 7) && aligned_to(w, 16) && aligned_to(q, 8) &&
        (!qt || (!(rows & 15) && !(ldqt & 15) && aligned_to(qt, 16)))) {
        launch_early(quant_blocks_vec_kernel, grid, 256, 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(w), ldw,
                     static_cast<__nv_fp8_storage_t*>(q), ldq, static_cast<__nv_fp8_storage_t*>(qt), ldqt, scale, scale_t, rows, cols);
        return cudaGetLastError() == cudaSuccess ? 0 : CAI_K_CUDA;
    }
    launch_early(quant_blocks_128x128_kernel, grid, 256, 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(w), ldw,
                 static_cast<__nv_fp8_storage_t*>(q), ldq, static_cast<__nv_fp8_storage_t*>(qt), ldqt, scale, scale_t, rows, cols);
    return cudaGetLastError() == cudaSuccess ? 0 : CAI_K_CUDA;
}
