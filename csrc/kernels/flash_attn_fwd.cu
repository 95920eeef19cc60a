// flash_attn_fwd.cu - causal grouped-query flash attention forward for sm_100a, head_dim 128.
//
// One CTA owns two adjacent 128-row query tiles (A and B) of one head and sweeps the key/value
// tiles they may attend to. Warp 0 streams Q, K and V tiles with TMA straight out of the packed
// QKV activation; warps 1 and 2 issue the tcgen05 MMAs of tile A and tile B (one issuer for both left a tile
// waiting behind the other's barriers: 6 x 640 tokens, 9 / 3 heads 28.5 -> 26.1 us, 8192 tokens, 32 / 8 heads
// 658 -> 618 us); warps 4-7 and 8-11 are the softmax groups of
// tile A and tile B, one thread per query row. Scores live in tensor memory: S = Q K^T lands in
// TMEM, the softmax group reads it with tcgen05.ld, writes the bf16 probabilities back over the
// same columns with tcgen05.st, and O += P V consumes P directly from TMEM as the A operand.
// While one group runs its softmax the tensor core works on the other tile, so the two overlap.
// The running maximum is only refreshed (and O rescaled in TMEM) when it grew by more than 2^8,
// which keeps that read-modify-write of O rare.
//
// TMEM map (512 columns): S_A/P_A 0-127, S_B/P_B 128-255, O_A 256-383, O_B 384-511.
//
// Replaces the one-thread-per-query kernel of the reference, which materialises the full
// [B, heads, T, T] probability tensor and has no GQA (src/cuda/cai_kernels.cu:80-109).
#include <math.h>

#include "cai_kernels.h"
#include "host_common.h"
#include "attn_common.cuh"
#include "sm100.cuh"

namespace cai {

constexpr int kAttnFwdThreads = 384;

struct AttnFwdParams {
    int B, S, nh, nkv;
    float scale_log2;
    __nv_bfloat16* out;
    float* lse;
    int* status;
};

// A warp's 32 finished rows of O, each lane with one: times `inv` to bf16, through 8 KB of the query tile, which nobody reads any more, so that the warp
// writes two whole rows at a time; from the registers every store met 32 lines. us, two CTAs to an SM,
// before / now: 8 x 384 tokens, 12 / 4 heads 14.8 / 11.9; 8 x 256, 32 / 8 17.2 / 15.6; 16 x 384, 16 / 4 27.7 / 25.2; 4 x 1024, 16 / 8 28.2 / 26.7.
__device__ __forceinline__ void put_out_rows(uint32_t stage, uint32_t tO, float inv, __nv_bfloat16* out, long long ld, int lane) {
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(tO + c * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int j4 = 0; j4 < 4; ++j4) {
            uint32_t o[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) o[t] = pack_bf16(__uint_as_float(v[j4 * 8 + 2 * t]) * inv, __uint_as_float(v[j4 * 8 + 2 * t + 1]) * inv);
            st_shared_v4(stage + lane * 256 + (((c * 4 + j4) ^ (lane & 7)) << 4), o[0], o[1], o[2], o[3]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int row = i * 2 + (lane >> 4), chunk = lane & 15;
        *reinterpret_cast<uint4*>(out + row * ld + chunk * 8) = ld_shared_v4(stage + row * 256 + ((chunk ^ (row & 7)) << 4));
    }
}

// Softmax of one query tile, whose scores arrive block by block in one buffer of tensor memory: one thread per query row (row r of
// the tile, lane bits in tS and tO), 128 threads. Ends by writing the tile's rows of the output.
__device__ __forceinline__ void softmax_tile(uint32_t tS, uint32_t tO, int r, int nx, uint64_t* s_full, uint64_t* p_full, uint64_t* o_final,
                                             volatile int* abort_flag, const AttnFwdParams& p, int b, int h, int row_base, int q0, const uint8_t* q_tile) {
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nx; ++j) {
        if (!mbar_wait_warp(s_full, j & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
        tc_fence_after();
        const bool diag = (j == nx - 1);
        // the whole score row (128 fp32) comes into registers with one wait and is used for both the
        // row maximum and the exponentials
        uint32_t sc[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + c * 32, sc[c]);
        tmem_ld_wait();
        float mx = -INFINITY;
        if (!diag) {
            float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                m0 = fmaxf(m0, __uint_as_float(sc[0][e]));
                m1 = fmaxf(m1, __uint_as_float(sc[1][e]));
                m2 = fmaxf(m2, __uint_as_float(sc[2][e]));
                m3 = fmaxf(m3, __uint_as_float(sc[3][e]));
            }
            mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int e = 0; e < 32; ++e)
                    if (c * 32 + e <= r) mx = fmaxf(mx, __uint_as_float(sc[c][e]));
        }
        const float m_new = fmaxf(m_used, mx * p.scale_log2);
        if (__any_sync(0xffffffffu, m_new > m_used + 8.f)) {
            const float alpha = fast_exp2(m_used - m_new);  // 0 on the first tile
            l *= alpha;
            if (j > 0) {
#pragma unroll 1
                for (int c = 0; c < 8; ++c) {   // sixteen columns at a time: the scores stay in registers meanwhile
                    uint32_t v[16];
                    tmem_ld_32x16(tO + c * 16, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
                    tmem_st_32x16(tO + c * 16, v);
                }
                tmem_st_wait();
            }
            m_used = m_new;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
            float l0 = 0.f, l1 = 0.f;
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
                float p0 = fast_exp2(fmaf(__uint_as_float(sc[c][e]), p.scale_log2, -m_used));
                float p1 = fast_exp2(fmaf(__uint_as_float(sc[c][e + 1]), p.scale_log2, -m_used));
                if (diag) {
                    if (c * 32 + e > r) p0 = 0.f;
                    if (c * 32 + e + 1 > r) p1 = 0.f;
                }
                l0 += p0;
                l1 += p1;
                pk[e >> 1] = pack_bf16(p0, p1);
            }
            l += l0 + l1;
            tmem_st_32x16(tS + c * 16, pk);
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive_warp(p_full);
    }
    if (ok && mbar_wait_warp(o_final, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) {
        tc_fence_after();
        const float inv = 1.f / l;
        const long long ldo = static_cast<long long>(p.nh) * kAttnHD;
        put_out_rows(smem_u32(q_tile) + (r >> 5) * 8192, tO, inv, p.out + (static_cast<long long>(row_base) + q0 + (r & ~31)) * ldo + h * kAttnHD, ldo, r & 31);
        if (p.lse)
            p.lse[(static_cast<long long>(b) * p.nh + h) * p.S + q0 + r] =
                (m_used + log2f(l)) * 0.6931471805599453f;
    }
}

__global__ void __launch_bounds__(kAttnFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm, const AttnFwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;                            // 2 tiles
    uint8_t* sK = smem + 2 * kAttnTileBytes;       // 2 stages
    uint8_t* sV = smem + 4 * kAttnTileBytes;       // 2 stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * kAttnTileBytes);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;
    uint64_t* k_empty = bars + 3;
    uint64_t* v_full = bars + 5;
    uint64_t* v_empty = bars + 7;
    uint64_t* s_full = bars + 9;
    uint64_t* p_full = bars + 11;
    uint64_t* o_final = bars + 13;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // CTAs are dispatched in linear block order; walk the query tiles slowest so that the heaviest
    // (latest) tiles of every head start first and the light ones fill the tail of the grid. (Pairing
    // tile i with tile last - i balances the CTAs but was slower: a step with one live tile costs as
    // much as a step with two.)
    const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    const int heads_all = gridDim.y * gridDim.z;
    const int pair = gridDim.x - 1 - lin / heads_all;
    const int h = (lin % heads_all) % gridDim.y, b = (lin % heads_all) / gridDim.y;
    const int g = h / (p.nh / p.nkv);
    const int qA = pair * 2 * kAttnTile, qB = qA + kAttnTile;
    const int nA = qA / kAttnTile + 1;
    const int nB = qB < p.S ? qB / kAttnTile + 1 : 0;
    const int n = nB > nA ? nB : nA;
    const int row_base = b * p.S;
    const int col_q = h * kAttnHD, col_k = (p.nh + g) * kAttnHD, col_v = (p.nh + p.nkv + g) * kAttnHD;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm);
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) {
            // both tiles' issuers hand a stage back. (Tile A, a key tile shorter, leaves the last one out: nobody waits for it.)
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], nB ? 2 : 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], nB ? 2 : 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);
            mbar_init(&o_final[i], 1);
        }
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

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer
            mbar_expect_tx(q_full, nB ? 2 * kAttnTileBytes : kAttnTileBytes);
            tma_load_2d(sQ, &tm, q_full, col_q, row_base + qA);
            tma_load_2d(sQ + kAttnSub, &tm, q_full, col_q + 64, row_base + qA);
            if (nB) {
                tma_load_2d(sQ + kAttnTileBytes, &tm, q_full, col_q, row_base + qB);
                tma_load_2d(sQ + kAttnTileBytes + kAttnSub, &tm, q_full, col_q + 64, row_base + qB);
            }
            bool ok = true;
            for (int j = 0; j < n && ok; ++j) {
                const int slot = j & 1;
                const uint32_t ph = (j >> 1) & 1;
                const int kv_row = row_base + j * kAttnTile;
                if (!mbar_wait(&k_empty[slot], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&k_full[slot], kAttnTileBytes);
                tma_load_2d(sK + slot * kAttnTileBytes, &tm, &k_full[slot], col_k, kv_row);
                tma_load_2d(sK + slot * kAttnTileBytes + kAttnSub, &tm, &k_full[slot], col_k + 64, kv_row);
                if (!mbar_wait(&v_empty[slot], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&v_full[slot], kAttnTileBytes);
                tma_load_2d(sV + slot * kAttnTileBytes, &tm, &v_full[slot], col_v, kv_row);
                tma_load_2d(sV + slot * kAttnTileBytes + kAttnSub, &tm, &v_full[slot], col_v + 64, kv_row);
            }
            grid_dep_launch();
            if (!ok)
                for (int i = 0; i < 32; ++i) __nanosleep(50000);
        }
    } else if (warp == 1 || warp == 2) {
        // ---------------- MMA issuers: warp 1 for tile A, warp 2 for tile B. The whole warp walks the loop (descriptors in
        // uniform registers), one lane issues. P is waited for last: the loads are normally there, so that P V(j) and
        // S(j+1) go out back to back once it arrives.
        const int X = warp - 1, nx = X ? nB : nA;
        const uint32_t idesc_qk = umma_idesc_bf16(128, 128, 0, 0), idesc_pv = umma_idesc_bf16(128, 128, 0, 1);
        const uint64_t qd = umma_smem_desc_sw128(smem_u32(sQ + X * kAttnTileBytes), 0, 1024);
        const uint64_t kd = umma_smem_desc_sw128(smem_u32(sK), 0, 1024), vd = umma_smem_desc_sw128(smem_u32(sV), kAttnSub, 1024);
        const uint32_t tS = tmem_base + X * 128, tO = tmem_base + 256 + X * 128;
        const bool leader = elect_one();
        if (nx > 0 && mbar_wait_warp(q_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) &&
            mbar_wait_warp(&k_full[0], 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) {
            tc_fence_after();
            if (leader) {
                issue_kk(tS, qd, kd, idesc_qk);
                umma_commit(&s_full[X]);
                umma_commit(&k_empty[0]);
            }
            for (int j = 0; j < nx; ++j) {
                const int slot = j & 1, ns = slot ^ 1;
                const bool more = j + 1 < nx;
                if (!mbar_wait_warp(&v_full[slot], (j >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                    (more && !mbar_wait_warp(&k_full[ns], ((j + 1) >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) ||
                    !mbar_wait_warp(&p_full[X], j & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN))
                    break;
                tc_fence_after();
                if (leader) {
                    issue_pv_desc(tO, tS, vd + slot * kTileDesc, idesc_pv, j > 0);
                    if (more) {
                        issue_kk(tS, qd, kd + ns * kTileDesc, idesc_qk);
                        umma_commit(&s_full[X]);
                        umma_commit(&k_empty[ns]);
                    } else {
                        umma_commit(&o_final[X]);
                    }
                    umma_commit(&v_empty[slot]);
                }
            }
        }
    } else if (warp >= 4) {
        // ---------------- softmax groups: warps 4-7 own tile A, warps 8-11 own tile B
        const int X = warp >= 8 ? 1 : 0;
        const int nx = X ? nB : nA;
        if (nx > 0) {
            const int r = (warp & 3) * 32 + lane;          // row inside the tile == TMEM lane
            const int q0 = X ? qB : qA;
            const uint32_t lane_bits = static_cast<uint32_t>((warp & 3) * 32) << 16;
            const uint32_t tS = tmem_base + X * 128 + lane_bits;
            const uint32_t tO = tmem_base + 256 + X * 128 + lane_bits;
            softmax_tile(tS, tO, r, nx, &s_full[X], &p_full[X], &o_final[X], abort_flag, p, b, h, row_base, q0, sQ + X * kAttnTileBytes);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}


// ---------------------------------------------------------------------------- one tile per CTA
// Variant for grids that do not fill the GPU (few heads per GPU under tensor parallelism), where the time is
// the critical path of the heaviest CTA. One CTA owns ONE query tile, the scores are double buffered in tensor
// memory and the MMA warp runs one key block ahead: S(j+1) = Q K(j+1)^T is issued before the softmax of block
// j has finished, so a step of the chain costs a softmax, not a softmax plus two MMAs plus two barrier round
// trips. O is rescaled only after the P V of the previous block has completed (barriers of its own, waited for in
// the rare rescale path and at the end).
//
// TMEM map: S0/P0 0-127, S1/P1 128-255, O 256-383.
constexpr int kAttnFwd1Threads = 256;

__global__ void __launch_bounds__(kAttnFwd1Threads, 1)
attn_fwd1_kernel(const __grid_constant__ CUtensorMap tm, const AttnFwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;
    uint8_t* sK = smem + 1 * kAttnTileBytes;       // 2 stages
    uint8_t* sV = smem + 3 * kAttnTileBytes;       // 2 stages
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 5 * kAttnTileBytes);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;
    uint64_t* k_empty = bars + 3;
    uint64_t* v_full = bars + 5;
    uint64_t* v_empty = bars + 7;
    uint64_t* s_full = bars + 9;    // [2] scores of a block are in S[b]
    uint64_t* p_full = bars + 11;   // [2] probabilities of a block are in S[b]
    // [2] P V of a block has completed (O may be touched), for even and for odd blocks. A warp that waits for block j - 1 has seen S(j), issued behind the
    // P V of block j - 2, and has not arrived for block j + 1: its barrier is in that phase or has just left it. (With a single barrier, waited for
    // behind the arrival for block j, the P V of block j could complete first; the parity of j - 1 was then that of a phase that
    // needed this warp's next arrival, and the CTA waited until its bound ran out.)
    uint64_t* pv_done = bars + 13;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    const int heads_all = gridDim.y * gridDim.z;
    const int tile = gridDim.x - 1 - lin / heads_all;   // heaviest (latest) query tiles of every head first
    const int h = (lin % heads_all) % gridDim.y, b = (lin % heads_all) / gridDim.y;
    const int g = h / (p.nh / p.nkv);
    const int q0 = tile * kAttnTile;
    const int n = tile + 1;                              // key blocks up to the diagonal
    const int row_base = b * p.S;
    const int col_q = h * kAttnHD, col_k = (p.nh + g) * kAttnHD, col_v = (p.nh + p.nkv + g) * kAttnHD;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm);
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);
        }
        mbar_init(&pv_done[0], 1);
        mbar_init(&pv_done[1], 1);
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

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(q_full, kAttnTileBytes);
            tma_load_2d(sQ, &tm, q_full, col_q, row_base + q0);
            tma_load_2d(sQ + kAttnSub, &tm, q_full, col_q + 64, row_base + q0);
            bool ok = true;
            for (int j = 0; j < n && ok; ++j) {
                const int slot = j & 1;
                const uint32_t ph = (j >> 1) & 1;
                const int kv_row = row_base + j * kAttnTile;
                if (!mbar_wait(&k_empty[slot], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&k_full[slot], kAttnTileBytes);
                tma_load_2d(sK + slot * kAttnTileBytes, &tm, &k_full[slot], col_k, kv_row);
                tma_load_2d(sK + slot * kAttnTileBytes + kAttnSub, &tm, &k_full[slot], col_k + 64, kv_row);
                if (!mbar_wait(&v_empty[slot], ph ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(&v_full[slot], kAttnTileBytes);
                tma_load_2d(sV + slot * kAttnTileBytes, &tm, &v_full[slot], col_v, kv_row);
                tma_load_2d(sV + slot * kAttnTileBytes + kAttnSub, &tm, &v_full[slot], col_v + 64, kv_row);
            }
            grid_dep_launch();
            if (!ok)
                for (int i = 0; i < 32; ++i) __nanosleep(50000);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc_qk = umma_idesc_bf16(128, 128, 0, 0);
            const uint32_t idesc_pv = umma_idesc_bf16(128, 128, 0, 1);
            const uint32_t sQa = smem_u32(sQ), sK0 = smem_u32(sK), sV0 = smem_u32(sV);
            const uint32_t tS[2] = {tmem_base, tmem_base + 128};
            const uint32_t tO = tmem_base + 256;
            bool ok = mbar_wait(q_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) &&
                      mbar_wait(&k_full[0], 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN);
            if (ok) {
                tc_fence_after();
                issue_qk(tS[0], sQa, sK0, idesc_qk);
                umma_commit(&s_full[0]);
                umma_commit(&k_empty[0]);
            }
            for (int j = 0; j < n && ok; ++j) {
                const int slot = j & 1;
                const uint32_t ph = (j >> 1) & 1;
                if (j + 1 < n) {
                    // one block ahead: S[(j+1)&1] last held P(j-1), whose P V was issued before this MMA
                    const int ns = (j + 1) & 1;
                    if (!mbar_wait(&k_full[ns], ((j + 1) >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                    tc_fence_after();
                    issue_qk(tS[ns], sQa, sK0 + ns * kAttnTileBytes, idesc_qk);
                    umma_commit(&s_full[ns]);
                    umma_commit(&k_empty[ns]);
                }
                if (!mbar_wait(&p_full[slot], ph, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                    !mbar_wait(&v_full[slot], ph, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                tc_fence_after();
                issue_pv(tO, tS[slot], sV0 + slot * kAttnTileBytes, idesc_pv, j > 0);
                umma_commit(&v_empty[slot]);
                umma_commit(&pv_done[slot]);
            }
        }
    } else if (warp >= 4) {
        const int r = (warp & 3) * 32 + lane;          // row inside the tile == TMEM lane
        const uint32_t lane_bits = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t tO = tmem_base + 256 + lane_bits;
        float m_used = -INFINITY, l = 0.f;
        bool ok = true;
        for (int j = 0; j < n; ++j) {
            const uint32_t tS = tmem_base + (j & 1) * 128 + lane_bits;
            if (!mbar_wait_warp(&s_full[j & 1], (j >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
            tc_fence_after();
            const bool diag = (j == n - 1);
            uint32_t sc[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + c * 32, sc[c]);
            tmem_ld_wait();
            float mx = -INFINITY;
            if (!diag) {
                float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    m0 = fmaxf(m0, __uint_as_float(sc[0][e]));
                    m1 = fmaxf(m1, __uint_as_float(sc[1][e]));
                    m2 = fmaxf(m2, __uint_as_float(sc[2][e]));
                    m3 = fmaxf(m3, __uint_as_float(sc[3][e]));
                }
                mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < 32; ++e)
                        if (c * 32 + e <= r) mx = fmaxf(mx, __uint_as_float(sc[c][e]));
            }
            const float m_new = fmaxf(m_used, mx * p.scale_log2);
            if (__any_sync(0xffffffffu, m_new > m_used + 8.f)) {
                const float alpha = fast_exp2(m_used - m_new);  // 0 on the first block
                l *= alpha;
                if (j > 0) {
                    // O is complete up to block j-1 only when that block's P V has finished
                    if (!mbar_wait_warp(&pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t v[32];
                        tmem_ld_32x32(tO + c * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
                        tmem_st_32x32(tO + c * 32, v);
                    }
                    tmem_st_wait();
                }
                m_used = m_new;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t pk[16];
                float l0 = 0.f, l1 = 0.f;
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    float p0 = fast_exp2(fmaf(__uint_as_float(sc[c][e]), p.scale_log2, -m_used));
                    float p1 = fast_exp2(fmaf(__uint_as_float(sc[c][e + 1]), p.scale_log2, -m_used));
                    if (diag) {
                        if (c * 32 + e > r) p0 = 0.f;
                        if (c * 32 + e + 1 > r) p1 = 0.f;
                    }
                    l0 += p0;
                    l1 += p1;
                    pk[e >> 1] = pack_bf16(p0, p1);
                }
                l += l0 + l1;
                tmem_st_32x16(tS + c * 16, pk);
            }
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive_warp(&p_full[j & 1]);
        }
        if (ok && mbar_wait_warp(&pv_done[(n - 1) & 1], ((n - 1) >> 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) {
            tc_fence_after();
            const float inv = 1.f / l;
            const long long ldo = static_cast<long long>(p.nh) * kAttnHD;
            put_out_rows(smem_u32(sQ) + (r >> 5) * 8192, tO, inv, p.out + (static_cast<long long>(row_base) + q0 + (r & ~31)) * ldo + h * kAttnHD, ldo, r & 31);
            if (p.lse)
                p.lse[(static_cast<long long>(b) * p.nh + h) * p.S + q0 + r] = (m_used + log2f(l)) * 0.6931471805599453f;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ---------------------------------------------------------------------------- two CTAs per SM
// One query tile per CTA, one buffer each for Q, K and V (96 KB) and for the scores (half of the tensor memory), so that two CTAs share
// an SM and each works while the other waits. What bounds a CTA with few
// key blocks is its own beginning and end (barriers, first loads, the output), which the other CTA of the SM now fills: 8 x 384 tokens, 12 / 4
// heads 19.7 -> 14.7 us against two tiles in one CTA.
// TMEM: S / P 0-127, O 128-255.
constexpr int kAttnHalfThreads = 192;   // warp 0 TMA, warp 1 MMA, warps 2-5 softmax

__global__ void __launch_bounds__(kAttnHalfThreads, 2)
attn_fwd_half_kernel(const __grid_constant__ CUtensorMap tm, const AttnFwdParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sQ = smem;
    uint8_t* sK = smem + 1 * kAttnTileBytes;
    uint8_t* sV = smem + 2 * kAttnTileBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 3 * kAttnTileBytes);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;
    uint64_t* k_empty = bars + 2;
    uint64_t* v_full = bars + 3;
    uint64_t* v_empty = bars + 4;
    uint64_t* s_full = bars + 5;
    uint64_t* o_final = bars + 6;
    uint64_t* p_full = bars + 7;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    const int heads_all = gridDim.y * gridDim.z;
    const int tile = gridDim.x - 1 - lin / heads_all;   // heaviest (latest) query tiles of every head first
    const int h = (lin % heads_all) % gridDim.y, b = (lin % heads_all) / gridDim.y;
    const int g = h / (p.nh / p.nkv);
    const int q0 = tile * kAttnTile;
    const int n = tile + 1;                              // key blocks up to the diagonal
    const int row_base = b * p.S;
    const int col_q = h * kAttnHD, col_k = (p.nh + g) * kAttnHD, col_v = (p.nh + p.nkv + g) * kAttnHD;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm);
        for (int i = 0; i < 7; ++i) mbar_init(&bars[i], 1);
        mbar_init(p_full, 4);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 256);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(q_full, kAttnTileBytes);
            tma_load_2d(sQ, &tm, q_full, col_q, row_base + q0);
            tma_load_2d(sQ + kAttnSub, &tm, q_full, col_q + 64, row_base + q0);
            bool ok = true;
            for (int j = 0; j < n && ok; ++j) {
                const int kv_row = row_base + j * kAttnTile;
                if (!mbar_wait(k_empty, (j & 1) ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(k_full, kAttnTileBytes);
                tma_load_2d(sK, &tm, k_full, col_k, kv_row);
                tma_load_2d(sK + kAttnSub, &tm, k_full, col_k + 64, kv_row);
                if (!mbar_wait(v_empty, (j & 1) ^ 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) { ok = false; break; }
                mbar_expect_tx(v_full, kAttnTileBytes);
                tma_load_2d(sV, &tm, v_full, col_v, kv_row);
                tma_load_2d(sV + kAttnSub, &tm, v_full, col_v + 64, kv_row);
            }
            grid_dep_launch();
            if (!ok)
                for (int i = 0; i < 32; ++i) __nanosleep(50000);
        }
    } else if (warp == 1) {
        const uint32_t idesc_qk = umma_idesc_bf16(128, 128, 0, 0), idesc_pv = umma_idesc_bf16(128, 128, 0, 1);
        const uint64_t qd = umma_smem_desc_sw128(smem_u32(sQ), 0, 1024), kd = umma_smem_desc_sw128(smem_u32(sK), 0, 1024);
        const uint64_t vd = umma_smem_desc_sw128(smem_u32(sV), kAttnSub, 1024);
        const uint32_t tS = tmem_base, tO = tmem_base + 128;
        const bool leader = elect_one();
        if (mbar_wait_warp(q_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) &&
            mbar_wait_warp(k_full, 0, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) {
            tc_fence_after();
            if (leader) {
                issue_kk(tS, qd, kd, idesc_qk);
                umma_commit(s_full);
                umma_commit(k_empty);
            }
            for (int j = 0; j < n; ++j) {
                const bool more = j + 1 < n;
                if (!mbar_wait_warp(v_full, j & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN) ||
                    (more && !mbar_wait_warp(k_full, (j + 1) & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN)) ||
                    !mbar_wait_warp(p_full, j & 1, abort_flag, p.status, CAI_DEV_TIMEOUT_ATTN))
                    break;
                tc_fence_after();
                if (leader) {
                    issue_pv_desc(tO, tS, vd, idesc_pv, j > 0);
                    umma_commit(v_empty);
                    if (more) {
                        issue_kk(tS, qd, kd, idesc_qk);
                        umma_commit(s_full);
                        umma_commit(k_empty);
                    } else {
                        umma_commit(o_final);
                    }
                }
            }
        }
    } else {
        const uint32_t lane_bits = static_cast<uint32_t>((warp & 3) * 32) << 16;
        softmax_tile(tmem_base + lane_bits, tmem_base + 128 + lane_bits, (warp & 3) * 32 + lane, n, s_full, p_full, o_final, abort_flag, p, b, h,
                     row_base, q0, sQ);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 256);
    }
}

}  // namespace cai

using namespace cai;

CAI_API int cai_flash_attn_fwd(const void* qkv, void* out, float* lse, int B, int S, int nh, int nkv, int hd,
                               float scale, void* stream) {
    return cai_flash_attn_fwd_variant(qkv, out, lse, B, S, nh, nkv, hd, scale, 0, stream);
}

// Grids that leave SMs idle (few heads per GPU) are bound by their heaviest CTA: one tile per CTA with the score MMA running a block
// ahead halves that path. Larger ones put two CTAs of one tile on each SM up to 4096 tokens, and two tiles in ping-pong into one
// CTA beyond, where both take the same time and the latter reads K and V half as often. All give the same bits. us, one tile / two tiles /
// two CTAs: 8 x 384 tokens, 12 / 4 heads 15.7 / 17.2 / 11.9; 6 x 640, 9 / 3 heads 17.7 / 17.1 / 15.0; 4 x 1024, 16 / 8 heads 40.7 / 31.9 /
// 26.7; 2048, 32 / 32 heads 61.0 / 46.7 / 45.7; 4 x 4096, 16 / 8 heads 388 / 309 / 306; 8192, 32 / 8 heads 721 / 490 / 544. In one wave of
// one-tile CTAs: 2 x 256, 16 / 8 7.2 / 8.3 / 7.4, 2048, 4 / 2 25.6 / 35.9 / 30.0.
// In between, one-tile CTAs overflow a wave. Up to three key tiles a wave of two-tile CTAs fills the SMs (256 tokens, 75 heads 11.6 / 9.2 / 8.9, 125 heads 14.0 /
// 10.1 / 10.8; 384, 50 heads 11.5 / 10.0 / 10.2, 70 heads 14.2 / 10.1 / 11.9). With more, the second wave of one-tile CTAs, the light ones, fits beside the
// heavy ones of the first until the sum of all steps holds it up, the later the more tiles a row has: from 1.25 CTAs an SM at 5 tiles, 1.6 at 8, 1.75 at 10 (one tile /
// two CTAs: 640 tokens, 33 heads 13.3 / 13.8, 42 heads 16.0 / 15.1; 1024, 25 heads 18.0 / 19.5, 34 heads 22.0 / 20.7; 1280, 20 heads 19.4 / 22.8, 29
// heads 25.5 / 24.4), and from 14 tiles on never within two waves (1792, 18 heads 27.5 / 31.1, 21 heads 31.4 / 31.6).
CAI_API int cai_flash_attn_fwd_form(int B, int S, int nh, int sms) {
    const long long tiles = S / kAttnTile, ctas = tiles * nh * B;
    if ((tiles + 1) / 2 * nh * B >= sms) return S <= 4096 ? 3 : 2;
    if (ctas <= sms) return 1;
    if (tiles <= 3) return 2;
    return tiles < 14 && 4 * tiles * ctas > sms * (9 * tiles - 20) ? 3 : 1;      // 2.25 - 5 / tiles CTAs an SM
}

CAI_API int cai_flash_attn_fwd_variant(const void* qkv, void* out, float* lse, int B, int S, int nh, int nkv, int hd,
                                       float scale, int force_variant, void* stream) {
    if (hd != kAttnHD || S % kAttnTile || nkv <= 0 || nh % nkv) {
        set_last_error("flash_attn_fwd: needs head_dim 128, seq %% 128 == 0, heads %% kv_heads == 0 (hd=%d S=%d)", hd, S);
        return CAI_K_BAD_ARG;
    }
    if (B <= 0 || S <= 0) return CAI_K_OK;
    const long long ld = static_cast<long long>(nh + 2 * nkv) * hd;
    CUtensorMap tm;
    if (!encode_tmap_2d(&tm, qkv, static_cast<uint64_t>(B) * S, ld, ld, 64, kAttnTile, 2)) return CAI_K_BAD_ARG;
    constexpr int smem_bytes = 6 * kAttnTileBytes + 1024 + 256;
    static bool configured[64] = {};
    const int dev = current_device();
    if (!configured[dev & 63]) {
        if (cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) !=
            cudaSuccess) {
            set_last_error("cudaFuncSetAttribute(attn_fwd) failed");
            return CAI_K_CUDA;
        }
        configured[dev & 63] = true;
    }
    AttnFwdParams p;
    p.B = B; p.S = S; p.nh = nh; p.nkv = nkv;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.out = static_cast<__nv_bfloat16*>(out);
    p.lse = lse;
    p.status = status_words(dev);
    const int variant = force_variant ? force_variant : cai_flash_attn_fwd_form(B, S, nh, sm_count(dev));
    if (variant == 3) {
        constexpr int smem_half = 3 * kAttnTileBytes + 1024 + 256;
        static bool configured_half[64] = {};
        if (!configured_half[dev & 63]) {
            if (cudaFuncSetAttribute(attn_fwd_half_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_half) != cudaSuccess ||
                cudaFuncSetAttribute(attn_fwd_half_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
                    cudaSuccess) {
                set_last_error("cudaFuncSetAttribute(attn_fwd_half) failed");
                return CAI_K_CUDA;
            }
            configured_half[dev & 63] = true;
        }
        launch_early(attn_fwd_half_kernel, dim3(S / kAttnTile, nh, B), kAttnHalfThreads, smem_half, static_cast<cudaStream_t>(stream), tm, p);
    } else if (variant == 1) {
        constexpr int smem1 = 5 * kAttnTileBytes + 1024 + 256;
        static bool configured1[64] = {};
        if (!configured1[dev & 63]) {
            if (cudaFuncSetAttribute(attn_fwd1_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1) != cudaSuccess) {
                set_last_error("cudaFuncSetAttribute(attn_fwd1) failed");
                return CAI_K_CUDA;
            }
            configured1[dev & 63] = true;
        }
        launch_early(attn_fwd1_kernel, dim3(S / kAttnTile, nh, B), kAttnFwd1Threads, smem1, static_cast<cudaStream_t>(stream), tm, p);
    } else {
        dim3 grid((S + 2 * kAttnTile - 1) / (2 * kAttnTile), nh, B);
        launch_early(attn_fwd_kernel, grid, kAttnFwdThreads, smem_bytes, static_cast<cudaStream_t>(stream), tm, p);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_last_error("attn_fwd launch failed: %s", cudaGetErrorString(e));
        return CAI_K_CUDA;
    }
    return CAI_K_OK;
}
