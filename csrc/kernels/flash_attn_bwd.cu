// flash_attn_bwd.cu - causal grouped-query flash attention backward for sm_100a, head_dim 128.
//
// Two launches, deterministic (no atomics):
//   1. attn_delta_kernel   delta[b,h,s] = sum_d dO * O                      (bandwidth bound)
//   2. attn_bwd_kernel, whose CTAs do one of two things:
//      dK / dV             one CTA per (kv tile, kv head, batch). It sweeps the query tiles at or
//                          below the diagonal of every query head of the group and accumulates
//                          dK and dV in tensor memory. Scores are computed transposed
//                          (S^T = K Q^T, dP^T = V dO^T) so that TMEM lanes are kv rows; the bf16
//                          P^T goes through shared memory and feeds dV += P^T dO from there, dS^T is
//                          written back over dP^T and feeds dK += dS^T Q as A operand straight from TMEM.
//      dQ                  one CTA per (q tile, head, batch): S = Q K^T, dP = dO V^T,
//                          dS -> TMEM, dQ += dS K.
// Q, K, V and dO tiles arrive by TMA from the packed activation; each shared-memory tile serves
// both as a K-major operand (for the score products) and as an MN-major operand (for the
// gradient products) through different UMMA descriptors, so nothing is transposed in memory.
//
// Roles per CTA: warp 0 issues TMA, warps 1 and 2 issue the MMAs, sixteen warps do the exponentials (four groups of
// four; a warp owns 32 TMEM lanes, a group 32 of the step's 128 score columns). What bounds a step is the latency chain
// of the compute warps, not the tensor pipe, so as little of that pipe's time as possible is left on the chain:
//   dK / dV: S^T(i+1) is computed as soon as the warps hold the scores of step i in registers. P^T leaves through shared
//            memory (in place of S^T it would hold up S^T(i+1) until dV(i) is done), before dP^T is looked at; dS^T goes
//            over dP^T in TMEM. Warp 1 issues S^T and dV, warp 2 dP^T and dK.
//   dQ:      warp 1 runs S ahead in two buffers, warp 2 alternates dP(j) and dQ(j).
// Two issuing warps because a wait costs the issuing thread 110-300 cycles even when it is already satisfied (its
// shared-memory access queues behind the operand reads of the MMAs): the other warp's MMAs run meanwhile. Each warp's MMAs
// execute in the order of issue, which is what protects dP / dS (one overwrites the other); the two warps share no
// operand that either writes. A thread keeps its 32 probabilities in fp32 registers until dP arrives. bf16 results in TMEM
// go over the first half of the 32 columns they came from, so the groups never touch each other's columns and need
// no barrier inside a step; a warp keeps the statistics of its queries in 32 words of its own. Every warp arrives once (not
// every thread) on a barrier. The softmax scale is applied once to the finished dK / dQ, and only diagonal tiles run the
// code path with the mask.
// Measured on a B200, before (one step at a time: scores, exponentials, gradients) and now, both back to back on one GPU:
// 8192 tokens, 32 / 8 heads: dK / dV 5390 -> 3700 cycles per 128 x 128 step and SM (1279 -> 1010 us: at 990 W the clock falls
// from 1900 to 1640 MHz), dQ 4240 -> 3030 cycles (986 -> 800 us). 4096 tokens, 16 / 8 heads: 203 -> 140 and 170 -> 111 us.
// P^T over S^T in TMEM, with S^T(i+1) behind dV(i): 8 % slower. Asking the barriers early without blocking, and fetching
// the next scores before dS^T is handed over: 2-10 % slower.
//
// Replaces the reference's one-thread-per-query backward, which recomputes dp twice, scatters
// dK/dV with atomicAdd and never zeroes dq/dk/dv (src/cuda/cai_kernels.cu:110-143).
#include <math.h>

#include "attn_common.cuh"
#include "cai_kernels.h"
#include "host_common.h"
#include "sm100.cuh"

namespace cai {

struct AttnBwdParams {
    int B, S, nh, nkv;
    float scale, scale_log2;
    const float* lse;
    const float* delta;
    __nv_bfloat16* dqkv;
    int* status;
    // dK / dV with one CTA per QUERY head (small grids): the heads of a kv group take turns adding their
    // contribution to the group's dK / dV rows; chain[b][g][kv tile] counts the heads that are done.
    int split_heads;
    unsigned int* chain;
    const float2* rope;          // (cos, sin) [S][64]: dQ and dK leave rotated back (null: as they are)
};

// chain counters of the head-split dK / dV kernel: one per (batch, kv group, kv tile).
// ONE array serves every call on a device: each call clears the slots it uses (in stream order: the row sums' kernel, or a
// memset) before its kernel, so two attention backwards that overlap on one GPU (different streams) would reset each other's
// counters. Calls that take the head-split path must therefore be ordered against each other; the executor
// issues them from one stream. A CTA of turn t waits (bounded) for the CTA of turn t - 1 of the same kv tile,
// which has a lower linear block id: with no more of these CTAs than SMs, and nothing beside them that waits, every one of them gets
// an SM whatever the order of dispatch; the launcher only takes this path then.
constexpr size_t kAttnChainSlots = 65536;
__device__ unsigned int g_attn_chain[kAttnChainSlots];

// Sixteen lanes per (token, head), 16 bytes a lane from each tensor, kDeltaUnroll of them in flight per thread: what bounds this is
// bytes in flight (one pair of 8-byte loads per thread and a 64-bit division in front: 8192 tokens of
// 32 heads 47 -> 23 us, 6 x 640 tokens of 9 heads 8.5 -> 6.2 us). The tensors are walked as one array of
// 128-element rows. (dO starts on 16 bytes, or its tensor map is refused; O may start on 8.)
constexpr int kDeltaUnroll = 2;
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ dout, float* __restrict__ delta,
                  unsigned total, unsigned S, unsigned nh, bool out16, unsigned int* chain, unsigned chain_slots) {
    grid_dep_begin();
    if (blockIdx.x * 256u + threadIdx.x < chain_slots) chain[blockIdx.x * 256u + threadIdx.x] = 0;   // for the dK / dV kernel behind this one
    const unsigned w0 = blockIdx.x * (16u * kDeltaUnroll) + (threadIdx.x >> 4);
    const int sub = threadIdx.x & 15;
    uint4 a[kDeltaUnroll], d[kDeltaUnroll];
#pragma unroll
    for (int i = 0; i < kDeltaUnroll; ++i) {
        const unsigned w = w0 + 16u * i;
        a[i] = d[i] = make_uint4(0, 0, 0, 0);
        if (w < total) {
            const size_t off = static_cast<size_t>(w) * kAttnHD + sub * 8;
            if (out16) {
                a[i] = *reinterpret_cast<const uint4*>(out + off);
            } else {
                const uint2 lo = *reinterpret_cast<const uint2*>(out + off), hi = *reinterpret_cast<const uint2*>(out + off + 4);
                a[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
            d[i] = *reinterpret_cast<const uint4*>(dout + off);
        }
    }
#pragma unroll
    for (int i = 0; i < kDeltaUnroll; ++i) {
        // two quads of elements per lane, added last: the tree of sums over quads 16, 8, 4, 2 and 1 apart
        float s0 = bf16_lo(a[i].x) * bf16_lo(d[i].x) + bf16_hi(a[i].x) * bf16_hi(d[i].x) + bf16_lo(a[i].y) * bf16_lo(d[i].y) +
                   bf16_hi(a[i].y) * bf16_hi(d[i].y);
        float s1 = bf16_lo(a[i].z) * bf16_lo(d[i].z) + bf16_hi(a[i].z) * bf16_hi(d[i].z) + bf16_lo(a[i].w) * bf16_lo(d[i].w) +
                   bf16_hi(a[i].w) * bf16_hi(d[i].w);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, o);
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        }
        const float s = s0 + s1;
        const unsigned w = w0 + 16u * i;
        if (sub == 0 && w < total) {
            const unsigned row = w / nh, h = w - row * nh, b = row / S, at = row - b * S;
            delta[(static_cast<size_t>(b) * nh + h) * S + at] = s;
        }
    }
}

// Sixteen compute warps: every scheduler has four of them to hide the TMEM and shared-memory latencies.
constexpr int kAttnGroups = 4;
constexpr int kAttnComputeThreads = kAttnGroups * 128;
constexpr int kAttnBwdThreads = 128 + kAttnComputeThreads;  // warp 0 TMA, warps 1-2 MMA, warps 4-19 compute

__device__ __forceinline__ void bar_sync_compute() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// A finished 128 x 128 fp32 accumulator goes to its bf16 rows through shared memory (operands nobody reads any more), so that a warp writes, and where
// it adds to what is there reads, two whole rows at a time. From the registers a lane had a row of its own, 32 lines an access: a turn of the heads' chain
// took 9 us, now 3.4. us, both parts and the row sums, before / now: 4 x 128 tokens, 2 / 1 heads 18.6 / 13.5; 512 tokens, 8 / 1 heads 75.4 / 40.2;
// 2048, 8 / 2 72.2 / 51.5; 8192, 2 / 1 138 / 124. (The old rows read ahead of every store, still a row per lane: no change.)
// Staged: row r at r * 512, its 16-byte chunk c at c ^ (r & 7).
__device__ __forceinline__ void stage_acc_chunk(uint32_t tacc, uint32_t stage, int r, int c) {
    uint32_t v[32];
    tmem_ld_32x32(tacc + c * 32, v);
    tmem_ld_wait();
#pragma unroll
    for (int k = 0; k < 8; ++k)
        st_shared_v4(stage + r * 512 + (((c * 8 + k) ^ (r & 7)) << 4), v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
}
// A thread of 512 takes kPieces times eight columns and the eight that are 64 further on: item `first` of eight a row, 128 rows a tile of 64 KB, then
// every 512th. Tile t leaves at dst[t], times mul[t]; where `rope` is given (the row of its table that belongs to row 0), tile 0 is rounded, as it
// would be in memory, and rotated back.
template <bool kAdd, int kPieces>
__device__ __forceinline__ void write_staged(uint32_t stage, __nv_bfloat16* const (&dst)[2], const float (&mul)[2], long long ld, int first, const float2* rope) {
    uint4 old[kPieces][2];
    if constexpr (kAdd) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int item = first + i * 512;
                old[i][h] = *reinterpret_cast<const uint4*>(dst[i >> 1] + ((item >> 3) & 127) * ld + h * 64 + (item & 7) * 8);
            }
    }
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
        const int item = first + i * 512, r = (item >> 3) & 127, c = (item & 7) * 2;
        const uint32_t row = stage + (i >> 1) * 65536 + r * 512;
        uint32_t o[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float4 f = ld_shared_f4(row + ((((h * 16) + c + k) ^ (r & 7)) << 4));
                v[4 * k] = f.x; v[4 * k + 1] = f.y; v[4 * k + 2] = f.z; v[4 * k + 3] = f.w;
            }
            const uint32_t ov[4] = {kAdd ? old[i][h].x : 0u, kAdd ? old[i][h].y : 0u, kAdd ? old[i][h].z : 0u, kAdd ? old[i][h].w : 0u};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                float lo = v[2 * t] * mul[i >> 1], hi = v[2 * t + 1] * mul[i >> 1];
                if constexpr (kAdd) {
                    lo += bf16_lo(ov[t]);
                    hi += bf16_hi(ov[t]);
                }
                o[h][t] = pack_bf16(lo, hi);
            }
        }
        if (rope && (i >> 1) == 0) {
            const float4* cs = reinterpret_cast<const float4*>(rope + r * 64 + (item & 7) * 8);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float4 q = cs[t];      // of two columns
                float a0 = bf16_lo(o[0][t]), a1 = bf16_hi(o[0][t]), b0 = bf16_lo(o[1][t]), b1 = bf16_hi(o[1][t]);
                rope_rotate(a0, b0, q.x, -q.y);
                rope_rotate(a1, b1, q.z, -q.w);
                o[0][t] = pack_bf16(a0, a1);
                o[1][t] = pack_bf16(b0, b1);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<uint4*>(dst[i >> 1] + r * ld + h * 64 + (item & 7) * 8) = make_uint4(o[h][0], o[h][1], o[h][2], o[h][3]);
    }
}

// Probabilities of one thread's 32 score columns, in place: exp2(s * scale_log2 - lse2). In the transposed form (dK / dV)
// a column is a query with its own lse2; in the other (dQ) the thread's row is the query. One half (16 columns) per call.
template <bool kDiag, int kHalf>
__device__ __forceinline__ void prob_cols(uint32_t (&v)[32], const float4 (&ls)[4], float scale_log2, int r, int qb) {
#pragma unroll
    for (int e4 = 0; e4 < 4; ++e4) {
        const float l[4] = {ls[e4].x, ls[e4].y, ls[e4].z, ls[e4].w};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int e = kHalf * 16 + e4 * 4 + t;
            float pv = fast_exp2(__uint_as_float(v[e]) * scale_log2 - l[t]);
            if constexpr (kDiag) {
                if (r > qb + e) pv = 0.f;  // key (row r) may not lie after the query (column)
            }
            v[e] = __float_as_uint(pv);
        }
    }
}
template <bool kDiag>
__device__ __forceinline__ void prob_rows(uint32_t (&v)[32], float lse2, float scale_log2, int r, int kb) {
#pragma unroll
    for (int e = 0; e < 32; ++e) {
        float pv = fast_exp2(__uint_as_float(v[e]) * scale_log2 - lse2);
        if constexpr (kDiag) {
            if (kb + e > r) pv = 0.f;
        }
        v[e] = __float_as_uint(pv);
    }
}

// D[128,hd] (+)= A[128,128](TMEM, bf16 pairs) * B[128,hd] with B MN-major in two 16 KiB sub-tiles; the A operand sits in
// four pieces of 16 columns, 32 columns apart (each where one warp group read its 32 fp32 columns from).
__device__ __forceinline__ void issue_pv_g16(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, bool accumulate) {
#pragma unroll
    for (int k = 0; k < kAttnTile / 16; ++k)
        umma_f16_ts(d_tmem, a_tmem + (k >> 1) * 32 + (k & 1) * 8, b_desc + k * (2048 >> 4), idesc, (accumulate || k > 0) ? 1u : 0u);
}
// D[128,hd] (+)= A[128,128] * B[128,hd], both in shared memory: A K-major, B MN-major.
__device__ __forceinline__ void issue_pd_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate) {
#pragma unroll
    for (int k = 0; k < kAttnTile / 16; ++k)
        umma_f16_ss(d_tmem, a_desc + (((k >> 2) * kAttnSub + (k & 3) * 32) >> 4), b_desc + k * (2048 >> 4), idesc,
                    (accumulate || k > 0) ? 1u : 0u);
}

// ---------------------------------------------------------------------------- dK / dV
// One CTA's work: number `lin` of the (kv tile, batch, head) triples.
__device__ __forceinline__ void attn_dkdv(const CUtensorMap& tm_qkv, const CUtensorMap& tm_do, const AttnBwdParams& p, uint8_t* smem, int lin) {
    uint8_t* sK = smem;
    uint8_t* sV = smem + kAttnTileBytes;
    uint8_t* sQ = smem + 2 * kAttnTileBytes;   // 2 stages
    uint8_t* sdO = smem + 4 * kAttnTileBytes;  // 2 stages
    uint8_t* sP = smem + 6 * kAttnTileBytes;   // P^T, the A operand of dV
    float* sStat = reinterpret_cast<float*>(smem + 7 * kAttnTileBytes);  // [16 warps][32] lse * log2e, later delta, of its columns
    uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + kAttnComputeThreads);
    uint64_t* kv_full = bars;
    uint64_t* q_full = bars + 1;      // [2]
    uint64_t* q_empty = bars + 3;     // [2] dK has read the tile (S^T long before)
    uint64_t* do_full = bars + 5;     // [2]
    uint64_t* do_empty = bars + 7;    // [2] dV and dP^T have read the tile
    uint64_t* s_full = bars + 9;
    uint64_t* s_empty = bars + 10;    // the compute warps have the scores in registers
    uint64_t* dp_full = bars + 11;
    uint64_t* p_ready = bars + 12;
    uint64_t* p_free = bars + 13;     // dV has read P^T
    uint64_t* ds_ready = bars + 14;
    uint64_t* final_bar = bars + 15;  // both issuing warps' last MMAs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // kv tile slowest, heaviest first; heads and batch fastest. Heads are kv groups (a CTA sweeps the group's query heads) or,
    // with split_heads, query heads
    const int heads = p.split_heads ? p.nh : p.nkv, heads_all = heads * p.B;
    const int j = lin / heads_all;  // kv tile
    const int ysel = (lin % heads_all) % heads, b = (lin % heads_all) / heads;
    const int rep = p.nh / p.nkv;
    const int g = p.split_heads ? ysel / rep : ysel;
    const int h_first = p.split_heads ? ysel : g * rep;
    const int turn = p.split_heads ? ysel - g * rep : 0;   // my place in the group's accumulation chain
    const int nq = p.S / kAttnTile;
    const int per_head = nq - j;          // query tiles at or below the diagonal
    const int iters = (p.split_heads ? 1 : rep) * per_head;
    const int row_base = b * p.S;
    const int col_k = (p.nh + g) * kAttnHD, col_v = (p.nh + p.nkv + g) * kAttnHD;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm_qkv);
        tma_prefetch_desc(&tm_do);
        mbar_init(kv_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&q_full[i], 1);
            mbar_init(&q_empty[i], 1);
            mbar_init(&do_full[i], 1);
            mbar_init(&do_empty[i], 2);
        }
        mbar_init(s_full, 1);
        mbar_init(s_empty, kAttnComputeThreads / 32);
        mbar_init(dp_full, 1);
        mbar_init(p_ready, kAttnComputeThreads / 32);
        mbar_init(p_free, 1);
        mbar_init(ds_ready, kAttnComputeThreads / 32);
        mbar_init(final_bar, 2);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 384;

    if (warp == 0) {
        if (lane == 0) {
            const int kv_row = row_base + j * kAttnTile;
            mbar_expect_tx(kv_full, 2 * kAttnTileBytes);
            tma_load_2d(sK, &tm_qkv, kv_full, col_k, kv_row);
            tma_load_2d(sK + kAttnSub, &tm_qkv, kv_full, col_k + 64, kv_row);
            tma_load_2d(sV, &tm_qkv, kv_full, col_v, kv_row);
            tma_load_2d(sV + kAttnSub, &tm_qkv, kv_full, col_v + 64, kv_row);
            bool ok = true;
            for (int it = 0; it < iters && ok; ++it) {
                const int slot = it & 1;
                const uint32_t ph = (it >> 1) & 1;
                const int h = h_first + it / per_head;
                const int q_row = row_base + (j + it % per_head) * kAttnTile;
                if (!mbar_wait(&q_empty[slot], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&q_full[slot], kAttnTileBytes);
                uint8_t* q = sQ + slot * kAttnTileBytes;
                tma_load_2d(q, &tm_qkv, &q_full[slot], h * kAttnHD, q_row);
                tma_load_2d(q + kAttnSub, &tm_qkv, &q_full[slot], h * kAttnHD + 64, q_row);
                if (!mbar_wait(&do_empty[slot], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&do_full[slot], kAttnTileBytes);
                uint8_t* d = sdO + slot * kAttnTileBytes;
                tma_load_2d(d, &tm_do, &do_full[slot], h * kAttnHD, q_row);
                tma_load_2d(d + kAttnSub, &tm_do, &do_full[slot], h * kAttnHD + 64, q_row);
            }
            grid_dep_launch();
            if (!ok)
                for (int i = 0; i < 32; ++i) __nanosleep(50000);
        }
    } else if (warp == 1) {
        // ---------------- S^T = K Q^T, a step ahead of the compute warps; dV += P^T dO. The whole warp walks the loop
        // (descriptors in uniform registers).
        const uint32_t idesc_kk = umma_idesc_bf16(128, 128, 0, 0), idesc_mn = umma_idesc_bf16(128, 128, 0, 1);
        const uint64_t kd = umma_smem_desc_sw128(smem_u32(sK), 0, 1024), qd = umma_smem_desc_sw128(smem_u32(sQ), 0, 1024);
        const uint64_t pd = umma_smem_desc_sw128(smem_u32(sP), 0, 1024), dod = umma_smem_desc_sw128(smem_u32(sdO), kAttnSub, 1024);
        const bool leader = elect_one();
        bool ok = mbar_wait_warp(kv_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN);
        for (int it = 0; it <= iters && ok; ++it) {
            if (it < iters) {
                const int slot = it & 1;
                if (!mbar_wait_warp(s_empty, (it & 1) ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                    !mbar_wait_warp(&q_full[slot], (it >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                tc_fence_after();
                if (leader) {
                    issue_kk(tS, kd, qd + slot * kTileDesc, idesc_kk);
                    umma_commit(s_full);
                }
            }
            if (it > 0) {
                const int slot = (it - 1) & 1;
                if (!mbar_wait_warp(&do_full[slot], ((it - 1) >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                    !mbar_wait_warp(p_ready, (it - 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                tc_fence_after();
                if (leader) {
                    issue_pd_ss(tdV, pd, dod + slot * kTileDesc, idesc_mn, it > 1);
                    umma_commit(p_free);
                    umma_commit(&do_empty[slot]);
                    if (it == iters) umma_commit(final_bar);
                }
            }
        }
    } else if (warp == 2) {
        // ---------------- dP^T = V dO^T, dK += dS^T Q (unscaled). dK(i) comes after S^T(i), which the compute warps saw before
        // they gave dS^T(i): the commit that frees Q(i) covers both its readers.
        const uint32_t idesc_kk = umma_idesc_bf16(128, 128, 0, 0), idesc_mn = umma_idesc_bf16(128, 128, 0, 1);
        const uint64_t vd = umma_smem_desc_sw128(smem_u32(sV), 0, 1024), dod = umma_smem_desc_sw128(smem_u32(sdO), 0, 1024);
        const uint64_t qd = umma_smem_desc_sw128(smem_u32(sQ), kAttnSub, 1024);
        const bool leader = elect_one();
        bool ok = mbar_wait_warp(kv_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN);
        for (int it = 0; it <= iters && ok; ++it) {
            if (it > 0) {
                const int slot = (it - 1) & 1;
                if (!mbar_wait_warp(&q_full[slot], ((it - 1) >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                    !mbar_wait_warp(ds_ready, (it - 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                tc_fence_after();
                if (leader) {
                    issue_pv_g16(tdK, tdP, qd + slot * kTileDesc, idesc_mn, it > 1);
                    umma_commit(&q_empty[slot]);
                    if (it == iters) umma_commit(final_bar);
                }
            }
            if (it < iters) {
                const int slot = it & 1;
                if (!mbar_wait_warp(&do_full[slot], (it >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                tc_fence_after();
                if (leader) {
                    issue_kk(tdP, vd, dod + slot * kTileDesc, idesc_kk);
                    umma_commit(dp_full);
                    umma_commit(&do_empty[slot]);
                }
            }
        }
    } else if (warp >= 4) {
        const int r = (warp & 3) * 32 + lane;  // kv row inside the tile == TMEM lane
        const int grp = (warp - 4) >> 2;       // which 32 of the step's 128 query columns
        const uint32_t lane_bits = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const int qb = grp * 32;               // first of this warp's 32 query columns
        const uint32_t tSg = tS + lane_bits + qb, tdPg = tdP + lane_bits + qb;
        float* stat = sStat + (warp - 4) * 32;
        // P^T row r, its 16-byte chunk c (8 queries) at chunk c ^ (r & 7) of the 128-byte row, 64 queries per sub-tile
        const uint32_t prow = smem_u32(sP) + (grp >> 1) * kAttnSub + r * 128;
        const uint32_t pchunk = (grp & 1) * 4, psw = r & 7;
        bool ok = true;
        // statistics of this warp's queries (a lane holds one), fetched a step ahead; shared through the warp's own 32 words
        auto stat_at = [&](const float* v, int it) {
            const int h = h_first + it / per_head;
            const int i = j + it % per_head;
            return v[(static_cast<long long>(b) * p.nh + h) * p.S + i * kAttnTile + qb + lane];
        };
        float lse_next = stat_at(p.lse, 0), delta_next = stat_at(p.delta, 0);
#pragma unroll 1
        for (int it = 0; it < iters; ++it) {
            const bool diag = it % per_head == 0;
            const float delta = delta_next;
            if (!mbar_wait_warp(s_full, it & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
            tc_fence_after();
            uint32_t pr[32];
            tmem_ld_32x32(tSg, pr);
            __syncwarp();
            stat[lane] = lse_next * 1.4426950408889634f;
            if (it + 1 < iters) {
                lse_next = stat_at(p.lse, it + 1);
                delta_next = stat_at(p.delta, it + 1);
            }
            __syncwarp();
            float4 ls[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) ls[e] = reinterpret_cast<const float4*>(stat)[e];
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive_warp(s_empty);
            if (diag) prob_cols<true, 0>(pr, ls, p.scale_log2, r, qb);
            else prob_cols<false, 0>(pr, ls, p.scale_log2, r, qb);
#pragma unroll
            for (int e = 0; e < 4; ++e) ls[e] = reinterpret_cast<const float4*>(stat)[4 + e];
            if (diag) prob_cols<true, 1>(pr, ls, p.scale_log2, r, qb);
            else prob_cols<false, 1>(pr, ls, p.scale_log2, r, qb);
            __syncwarp();
            stat[lane] = delta;
            if (it > 0 && !mbar_wait_warp(p_free, (it - 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
            auto give_p = [&]() {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t o[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        o[t] = pack_bf16(__uint_as_float(pr[c * 8 + 2 * t]), __uint_as_float(pr[c * 8 + 2 * t + 1]));
                    st_shared_v4(prow + (((pchunk + c) ^ psw) << 4), o[0], o[1], o[2], o[3]);
                }
                fence_proxy_async_smem();
                mbar_arrive_warp(p_ready);
            };
            give_p();
            if (!mbar_wait_warp(dp_full, it & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
            tc_fence_after();
            uint32_t dp[32];
            tmem_ld_32x32(tdPg, dp);
            tmem_ld_wait();
            uint32_t dk[16];
#pragma unroll
            for (int e4 = 0; e4 < 8; ++e4) {
                const float4 d = reinterpret_cast<const float4*>(stat)[e4];
                const int e = e4 * 4;
                dk[e4 * 2] = pack_bf16(__uint_as_float(pr[e]) * (__uint_as_float(dp[e]) - d.x),
                                       __uint_as_float(pr[e + 1]) * (__uint_as_float(dp[e + 1]) - d.y));
                dk[e4 * 2 + 1] = pack_bf16(__uint_as_float(pr[e + 2]) * (__uint_as_float(dp[e + 2]) - d.z),
                                           __uint_as_float(pr[e + 3]) * (__uint_as_float(dp[e + 3]) - d.w));
            }
            tmem_st_32x16(tdPg, dk);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive_warp(ds_ready);
        }
        // every MMA of the tile is done, and with it every read of shared memory; groups 0, 1 stage dK, 2, 3 dV. A warp that gave up comes to the
        // barriers all the same.
        ok = ok && mbar_wait_warp(final_bar, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN);
        const uint32_t stage = smem_u32(smem);
        if (ok) {
            tc_fence_after();
            const int c0 = (grp & 1) * 2;
            stage_acc_chunk((grp < 2 ? tdK : tdV) + lane_bits, stage + (grp >> 1) * 65536, r, c0);
            stage_acc_chunk((grp < 2 ? tdK : tdV) + lane_bits, stage + (grp >> 1) * 65536, r, c0 + 1);
        }
        bar_sync_compute();
        const long long ld = static_cast<long long>(p.nh + 2 * p.nkv) * kAttnHD;
        __nv_bfloat16* row0 = p.dqkv + (static_cast<long long>(row_base) + j * kAttnTile) * ld;
        __nv_bfloat16* const dst[2] = {row0 + col_k, row0 + col_v};
        const float mul[2] = {p.scale, 1.f};
        const int first = threadIdx.x - 128;
        unsigned int* cnt = p.split_heads ? p.chain + (static_cast<long long>(b) * p.nkv + g) * nq + j : nullptr;
        if (turn > 0 && ok) {
            // heads of the group add in turn: wait (bounded) until the heads before me are done
            ok = false;
            for (uint32_t spin = 0; spin < kSpinLimit && !ok; ++spin) {
                unsigned int v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
                ok = v >= static_cast<unsigned int>(turn);
                if (!ok && spin > 16) __nanosleep(200);
            }
            if (!ok) atomicCAS(p.status, 0, CAI_DEV_TIMEOUT_ATTN);
        }
        if (ok) {
            // the last of the heads turns the finished sum
            const float2* rope = p.rope && (!p.split_heads || turn + 1 == rep) ? p.rope + static_cast<long long>(j) * kAttnTile * 64 : nullptr;
            if (turn == 0) write_staged<false, 4>(stage, dst, mul, ld, first, rope);
            else write_staged<true, 4>(stage, dst, mul, ld, first, rope);
        }
        if (p.split_heads) {
            __threadfence();
            bar_sync_compute();
            if (threadIdx.x == 128) {   // first compute thread: everyone's rows are written and fenced
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(cnt), "r"(static_cast<unsigned int>(turn + 1)) : "memory");
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ---------------------------------------------------------------------------- dQ
__device__ __forceinline__ void attn_dq(const CUtensorMap& tm_qkv, const CUtensorMap& tm_do, const AttnBwdParams& p, uint8_t* smem, int lin) {
    uint8_t* sQ = smem;
    uint8_t* sdO = smem + kAttnTileBytes;
    uint8_t* sK = smem + 2 * kAttnTileBytes;  // 3 stages: S runs a step ahead of the dQ that still needs the tile
    uint8_t* sV = smem + 5 * kAttnTileBytes;  // 2 stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 7 * kAttnTileBytes);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;     // [3]
    uint64_t* k_empty = bars + 4;    // [3] dQ has read the tile
    uint64_t* v_full = bars + 7;     // [2]
    uint64_t* v_empty = bars + 9;    // [2]
    uint64_t* s_full = bars + 11;    // [2]
    uint64_t* s_empty = bars + 13;   // [2] the compute warps have read the scores
    uint64_t* dp_full = bars + 15;
    uint64_t* ds_ready = bars + 16;
    uint64_t* final_bar = bars + 17;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int heads_all = p.nh * p.B;
    const int i = p.S / kAttnTile - 1 - lin / heads_all;  // q tile, heaviest first across all heads
    const int h = (lin % heads_all) % p.nh, b = (lin % heads_all) / p.nh;
    const int g = h / (p.nh / p.nkv);
    const int n = i + 1;
    const int row_base = b * p.S;
    const int col_q = h * kAttnHD, col_k = (p.nh + g) * kAttnHD, col_v = (p.nh + p.nkv + g) * kAttnHD;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm_qkv);
        tma_prefetch_desc(&tm_do);
        mbar_init(q_full, 1);
        for (int k = 0; k < 3; ++k) {
            mbar_init(&k_full[k], 1);
            mbar_init(&k_empty[k], 1);
        }
        for (int k = 0; k < 2; ++k) {
            mbar_init(&v_full[k], 1);
            mbar_init(&v_empty[k], 1);
            mbar_init(&s_full[k], 1);
            mbar_init(&s_empty[k], kAttnComputeThreads / 32);
        }
        mbar_init(dp_full, 1);
        mbar_init(ds_ready, kAttnComputeThreads / 32);
        mbar_init(final_bar, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tdP = tmem_base + 256, tdQ = tmem_base + 384;   // two score buffers

    if (warp == 0) {
        if (lane == 0) {
            const int q_row = row_base + i * kAttnTile;
            mbar_expect_tx(q_full, 2 * kAttnTileBytes);
            tma_load_2d(sQ, &tm_qkv, q_full, col_q, q_row);
            tma_load_2d(sQ + kAttnSub, &tm_qkv, q_full, col_q + 64, q_row);
            tma_load_2d(sdO, &tm_do, q_full, col_q, q_row);
            tma_load_2d(sdO + kAttnSub, &tm_do, q_full, col_q + 64, q_row);
            bool ok = true;
            int ks = 0;
            uint32_t kph = 0;
            for (int j = 0; j < n && ok; ++j) {
                const int slot = j & 1;
                const uint32_t ph = (j >> 1) & 1;
                const int kv_row = row_base + j * kAttnTile;
                if (!mbar_wait(&k_empty[ks], kph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&k_full[ks], kAttnTileBytes);
                uint8_t* k = sK + ks * kAttnTileBytes;
                tma_load_2d(k, &tm_qkv, &k_full[ks], col_k, kv_row);
                tma_load_2d(k + kAttnSub, &tm_qkv, &k_full[ks], col_k + 64, kv_row);
                if (!mbar_wait(&v_empty[slot], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&v_full[slot], kAttnTileBytes);
                uint8_t* v = sV + slot * kAttnTileBytes;
                tma_load_2d(v, &tm_qkv, &v_full[slot], col_v, kv_row);
                tma_load_2d(v + kAttnSub, &tm_qkv, &v_full[slot], col_v + 64, kv_row);
                if (++ks == 3) {
                    ks = 0;
                    kph ^= 1;
                }
            }
            grid_dep_launch();
            if (!ok)
                for (int k = 0; k < 32; ++k) __nanosleep(50000);
        }
    } else if (warp == 1) {
        // ---------------- S = Q K^T, up to two steps ahead of the compute warps
        const uint32_t idesc_kk = umma_idesc_bf16(128, 128, 0, 0);
        const uint64_t qd = umma_smem_desc_sw128(smem_u32(sQ), 0, 1024), kd = umma_smem_desc_sw128(smem_u32(sK), 0, 1024);
        const bool leader = elect_one();
        bool ok = mbar_wait_warp(q_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN);
        int ks = 0;
        uint32_t kph = 0;
        for (int j = 0; j < n && ok; ++j) {
            const int buf = j & 1;
            if (!mbar_wait_warp(&k_full[ks], kph, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                !mbar_wait_warp(&s_empty[buf], ((j >> 1) & 1) ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
            tc_fence_after();
            if (leader) {
                issue_kk(tS + buf * 128, qd, kd + ks * kTileDesc, idesc_kk);
                umma_commit(&s_full[buf]);
            }
            if (++ks == 3) {
                ks = 0;
                kph ^= 1;
            }
        }
    } else if (warp == 2) {
        // ---------------- dP = dO V^T, dQ += dS K (unscaled). Ordered behind S(j) by ds_ready(j), which the compute warps
        // give after they have seen S(j): the commit that frees K(j) therefore covers both its readers.
        const uint32_t idesc_kk = umma_idesc_bf16(128, 128, 0, 0), idesc_mn = umma_idesc_bf16(128, 128, 0, 1);
        const uint64_t dod = umma_smem_desc_sw128(smem_u32(sdO), 0, 1024), vd = umma_smem_desc_sw128(smem_u32(sV), 0, 1024);
        const uint64_t kd = umma_smem_desc_sw128(smem_u32(sK), kAttnSub, 1024);
        const bool leader = elect_one();
        bool ok = mbar_wait_warp(q_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN);
        int ks = 0;            // ring slot and phase of the K tile of step j - 1
        uint32_t kph = 0;
        for (int j = 0; j <= n && ok; ++j) {
            const int slot = j & 1;
            if (j > 0) {
                if (!mbar_wait_warp(&k_full[ks], kph, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                    !mbar_wait_warp(ds_ready, (j - 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                tc_fence_after();
                if (leader) {
                    issue_pv_g16(tdQ, tdP, kd + ks * kTileDesc, idesc_mn, j > 1);
                    umma_commit(&k_empty[ks]);
                    if (j == n) umma_commit(final_bar);
                }
                if (++ks == 3) {
                    ks = 0;
                    kph ^= 1;
                }
            }
            if (j < n) {
                if (!mbar_wait_warp(&v_full[slot], (j >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                tc_fence_after();
                if (leader) {
                    issue_kk(tdP, dod, vd + slot * kTileDesc, idesc_kk);
                    umma_commit(dp_full);
                    umma_commit(&v_empty[slot]);
                }
            }
        }
    } else if (warp >= 4) {
        const int r = (warp & 3) * 32 + lane;  // q row inside the tile
        const int grp = (warp - 4) >> 2;       // which 32 of the step's 128 key columns
        const uint32_t lane_bits = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const long long vec = (static_cast<long long>(b) * p.nh + h) * p.S + i * kAttnTile + r;
        const float lse2 = p.lse[vec] * 1.4426950408889634f;
        const float dl = p.delta[vec];
        const int kb = grp * 32;   // first of this warp's 32 key columns
        const uint32_t tdPg = tdP + lane_bits + kb;
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < n; ++j) {
            const int buf = j & 1;
            if (!mbar_wait_warp(&s_full[buf], (j >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
            tc_fence_after();
            uint32_t pr[32];
            tmem_ld_32x32(tS + buf * 128 + lane_bits + kb, pr);
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive_warp(&s_empty[buf]);
            if (j == i) prob_rows<true>(pr, lse2, p.scale_log2, r, kb);
            else prob_rows<false>(pr, lse2, p.scale_log2, r, kb);
            if (!mbar_wait_warp(dp_full, j & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
            tc_fence_after();
            uint32_t dp[32], dk[16];
            tmem_ld_32x32(tdPg, dp);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; e += 2)
                dk[e >> 1] = pack_bf16(__uint_as_float(pr[e]) * (__uint_as_float(dp[e]) - dl),
                                       __uint_as_float(pr[e + 1]) * (__uint_as_float(dp[e + 1]) - dl));
            tmem_st_32x16(tdPg, dk);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive_warp(ds_ready);
        }
        ok = ok && mbar_wait_warp(final_bar, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN);
        const uint32_t stage = smem_u32(smem);
        if (ok) {
            tc_fence_after();
            stage_acc_chunk(tdQ + lane_bits, stage, r, grp);
        }
        bar_sync_compute();
        if (ok) {
            const long long ld = static_cast<long long>(p.nh + 2 * p.nkv) * kAttnHD;
            __nv_bfloat16* dst0 = p.dqkv + (static_cast<long long>(row_base) + i * kAttnTile) * ld + col_q;
            __nv_bfloat16* const dst[2] = {dst0, nullptr};
            const float mul[2] = {p.scale, 0.f};
            write_staged<false, 2>(stage, dst, mul, ld, threadIdx.x - 128, p.rope ? p.rope + static_cast<long long>(i) * kAttnTile * 64 : nullptr);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ---------------------------------------------------------------------------- both
// The first `dkdv_ctas` CTAs work on dK / dV, the others on dQ: the two need the same set-up, shared memory and registers, and neither reads
// what the other writes. As launches of their own each ended in a wave that leaves SMs idle, and a dK / dV part of few kv heads leaves
// them idle throughout; together the light CTAs of one fill up behind the heavy ones of the other. Forward, backward and both rotary embeddings, two
// launches and one: 8 x 384 tokens, 12 / 4 heads (96 and 288 CTAs) 73.9 -> 65.4 us; 7 x 256, 4 / 2 heads 45.3 -> 41.9; 3 x 2432, 32 / 8 heads
// 854 -> 837; 8192 tokens, 32 / 8 heads 2504 -> 2466. A chain of split heads (AttnBwdParams) waits only for CTAs of lower number, and dQ's CTAs wait
// for nobody: they leave their SMs to whatever part of the chain is not there yet.
__global__ void __launch_bounds__(kAttnBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do, const AttnBwdParams p,
                const int dkdv_ctas) {
    // no room to round the base up: tiles start on swizzle boundaries only if the shared window does (checked)
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023) {
        grid_dep_wait();
        if (threadIdx.x == 0) atomicCAS(p.status, 0, CAI_DEV_BAD_ARG);
        return;
    }
    const int cta = static_cast<int>(blockIdx.x);
    if (cta < dkdv_ctas) attn_dkdv(tm_qkv, tm_do, p, smem, cta);
    else attn_dq(tm_qkv, tm_do, p, smem, cta - dkdv_ctas);
}

}  // namespace cai

using namespace cai;

CAI_API int cai_flash_attn_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* delta,
                               void* dqkv, int B, int S, int nh, int nkv, int hd, float scale, void* stream) {
    return cai_flash_attn_bwd_parts(qkv, out, dout, lse, delta, dqkv, B, S, nh, nkv, hd, scale, 7, stream);
}

CAI_API int cai_flash_attn_bwd_parts(const void* qkv, const void* out, const void* dout, const float* lse, float* delta,
                                     void* dqkv, int B, int S, int nh, int nkv, int hd, float scale, int parts, void* stream) {
    return cai_flash_attn_bwd_rope(qkv, out, dout, lse, delta, dqkv, nullptr, B, S, nh, nkv, hd, scale, parts, stream);
}

CAI_API int cai_flash_attn_bwd_rope(const void* qkv, const void* out, const void* dout, const float* lse, float* delta, void* dqkv,
                                    const float* table, int B, int S, int nh, int nkv, int hd, float scale, int parts, void* stream) {
    if (hd != kAttnHD || S % kAttnTile || nkv <= 0 || nh % nkv) {
        set_last_error("flash_attn_bwd: needs head_dim 128, seq %% 128 == 0, heads %% kv_heads == 0");
        return CAI_K_BAD_ARG;
    }
    if (B <= 0 || S <= 0) return CAI_K_OK;
    if (reinterpret_cast<uintptr_t>(table) & 15) {
        set_last_error("flash_attn_bwd: the rotary table must start on 16 bytes");
        return CAI_K_BAD_ARG;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long ld = static_cast<long long>(nh + 2 * nkv) * hd;
    const long long ldo = static_cast<long long>(nh) * hd;
    CUtensorMap tm_qkv, tm_do;
    if (!encode_tmap_2d(&tm_qkv, qkv, static_cast<uint64_t>(B) * S, ld, ld, 64, kAttnTile, 2)) return CAI_K_BAD_ARG;
    if (!encode_tmap_2d(&tm_do, dout, static_cast<uint64_t>(B) * S, ldo, ldo, 64, kAttnTile, 2)) return CAI_K_BAD_ARG;
    constexpr int smem_bytes = 7 * kAttnTileBytes + 2048 + 256;
    static bool configured[64] = {};
    const int dev = current_device();
    if (!configured[dev & 63]) {
        if (cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) {
            set_last_error("cudaFuncSetAttribute(attn_bwd) failed");
            return CAI_K_CUDA;
        }
        configured[dev & 63] = true;
    }
    AttnBwdParams p;
    p.B = B; p.S = S; p.nh = nh; p.nkv = nkv;
    p.scale = scale;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.lse = lse;
    p.delta = delta;
    p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
    p.status = status_words(dev);
    const int nq = S / kAttnTile;
    // Few kv groups per GPU (tensor parallelism): one CTA per query head instead of per kv group shortens the
    // longest CTA by the group size; the heads of a group then add into dK / dV in turn (chain counters).
    p.split_heads = 0;
    p.chain = nullptr;
    p.rope = reinterpret_cast<const float2*>(table);
    const size_t need = static_cast<size_t>(B) * nkv * nq;
    if ((parts & 2) && nh > nkv && static_cast<long long>(nq) * nkv * B < sm_count(dev) &&
        static_cast<long long>(nq) * nh * B <= sm_count(dev) && need <= kAttnChainSlots) {
        // the counters live in a device array of the library: nothing is allocated on this path. The first call
        // on a device resolves the array's address (which may load the module), so it should come before any
        // stream capture; later calls only enqueue work.
        static unsigned int* chain_ptr[64] = {};
        if (!chain_ptr[dev & 63] &&
            cudaGetSymbolAddress(reinterpret_cast<void**>(&chain_ptr[dev & 63]), g_attn_chain) != cudaSuccess) {
            set_last_error("attn_bwd: cannot resolve the chain counters");
            return CAI_K_CUDA;
        }
        // the row sums' kernel clears the slots where it runs first (it has 8 threads for each row of a head, a slot is 128 rows)
        if (!(parts & 1) && cudaMemsetAsync(chain_ptr[dev & 63], 0, need * sizeof(unsigned int), st) != cudaSuccess) return CAI_K_CUDA;
        p.split_heads = 1;
        p.chain = chain_ptr[dev & 63];
    }
    const long long rows = static_cast<long long>(B) * S * nh;
    if (parts & 1) {
        constexpr unsigned per_cta = 16u * kDeltaUnroll;
        launch_early(attn_delta_kernel, static_cast<unsigned>((rows + per_cta - 1) / per_cta), 256, 0, st,
                     static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(dout), delta, static_cast<unsigned>(rows),
                     static_cast<unsigned>(S), static_cast<unsigned>(nh), (reinterpret_cast<uintptr_t>(out) & 15) == 0, p.chain,
                     static_cast<unsigned>(p.split_heads ? need : 0));
    }
    const long long kv_ctas = (parts & 2) ? static_cast<long long>(nq) * (p.split_heads ? nh : nkv) * B : 0;
    const long long q_ctas = (parts & 4) ? static_cast<long long>(nq) * nh * B : 0;
    if (kv_ctas + q_ctas)
        launch_early(attn_bwd_kernel, static_cast<unsigned>(kv_ctas + q_ctas), kAttnBwdThreads, smem_bytes, st, tm_qkv, tm_do, p,
                     static_cast<int>(kv_ctas));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_last_error("attn_bwd launch failed: %s", cudaGetErrorString(e));
        return CAI_K_CUDA;
    }
    return CAI_K_OK;
}
