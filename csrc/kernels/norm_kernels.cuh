// norm_kernels.cuh - device code of RMSNorm backward, shared by the two translation units that
// launch it (pointwise.cu and rmsnorm_bwd_static.cu), plus the small vector / reduction helpers the
// bandwidth-bound kernels use. Kernels are `static` so that each including file owns its copy.
#pragma once

#include <math.h>

#include "host_common.h"
#include "norm_form.h"
#include "sm100.cuh"

namespace cai {

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
    f[0] = bf16_lo(v.x); f[1] = bf16_hi(v.x);
    f[2] = bf16_lo(v.y); f[3] = bf16_hi(v.y);
    f[4] = bf16_lo(v.z); f[5] = bf16_hi(v.z);
    f[6] = bf16_lo(v.w); f[7] = bf16_hi(v.w);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint4 o;
    o.x = pack_bf16(f[0], f[1]);
    o.y = pack_bf16(f[2], f[3]);
    o.z = pack_bf16(f[4], f[5]);
    o.w = pack_bf16(f[6], f[7]);
    return o;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// Sum over the block; every thread gets the result. `red` is >= 33 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        float t = lane < nw ? red[lane] : 0.f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}
__device__ __forceinline__ float block_max(float v, float* red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        float t = lane < nw ? red[lane] : -INFINITY;
        t = warp_max(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

constexpr int kNormThreads = 256;
constexpr int kNormWarpCols = 2048;  // columns one warp covers: 32 lanes x 8 chunks x 8 elements

// Backward, input gradient: dx (+)= rr * dy * g - rr^3 * x * sum(dy * g * x) / H. A row is handled
// by R = ceil(H / 2048) warps that keep their slice of x and dy in registers (each tensor is read
// once); a CTA of 8 warps works on 8 / R rows at a time.
static __global__ void __launch_bounds__(kNormThreads)
rmsnorm_bwd_dx_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ g,
                      const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ dy,
                      __nv_bfloat16* __restrict__ dx, int rows, int H, int dx_acc, int R) {
    grid_dep_begin();
    __shared__ float part[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = 8 / R;
    const int grp = warp / R, sub = warp - grp * R;
    const bool active = grp < groups;
    const int col0 = sub * kNormWarpCols;
    const uint4* gr = reinterpret_cast<const uint4*>(g);
    for (long long base = static_cast<long long>(blockIdx.x) * groups; base < rows; base += static_cast<long long>(gridDim.x) * groups) {
        const long long row = base + grp;
        const bool live = active && row < rows;
        uint4 xv[8], dv[8];
        float S = 0.f;
        if (live) {
            const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
            const uint4* dyr = reinterpret_cast<const uint4*>(dy + row * H);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int col = col0 + (c * 32 + lane) * 8;
                if (col < H) {
                    xv[c] = xr[col >> 3];
                    dv[c] = dyr[col >> 3];
                }
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int col = col0 + (c * 32 + lane) * 8;
                if (col < H) {
                    float xf[8], df[8], gf[8];
                    unpack8(xv[c], xf);
                    unpack8(dv[c], df);
                    unpack8(gr[col >> 3], gf);
#pragma unroll
                    for (int e = 0; e < 8; ++e) S += df[e] * gf[e] * xf[e];
                }
            }
        }
        S = warp_sum(S);
        if (R > 1) {
            if (lane == 0) part[warp] = S;
            __syncthreads();
            if (active) {
                S = 0.f;
                for (int k = 0; k < R; ++k) S += part[grp * R + k];
            }
            __syncthreads();
        }
        if (live) {
            const float rr = rstd[row];
            const float k3 = rr * rr * rr * S / H;
            uint4* dxr = reinterpret_cast<uint4*>(dx + row * H);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int col = col0 + (c * 32 + lane) * 8;
                if (col < H) {
                    float xf[8], df[8], gf[8], o[8];
                    unpack8(xv[c], xf);
                    unpack8(dv[c], df);
                    unpack8(gr[col >> 3], gf);
                    if (dx_acc) unpack8(dxr[col >> 3], o);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float v = rr * df[e] * gf[e] - k3 * xf[e];
                        o[e] = dx_acc ? o[e] + v : v;
                    }
                    dxr[col >> 3] = pack8(o);
                }
            }
        }
    }
}

// Backward, gain gradient: partial[part][col] = sum over the part's rows of dy * x * rstd. Threads
// own columns (coalesced 16-byte loads), CTAs own row ranges; x and dy were just streamed by the dx
// kernel, so this second sweep is mostly served from L2.
static __global__ void __launch_bounds__(256)
rmsnorm_bwd_dg_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ rstd,
                      const __nv_bfloat16* __restrict__ dy, float* __restrict__ dg_partial, int rows, int H,
                      int rows_per_part) {
    grid_dep_begin();
    const long long r0 = static_cast<long long>(blockIdx.x) * rows_per_part;
    const long long r1 = r0 + rows_per_part < rows ? r0 + rows_per_part : rows;
    for (int c = threadIdx.x; c < (H >> 3); c += 256) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (long long r = r0; r < r1; ++r) {
            float xf[8], df[8];
            unpack8(reinterpret_cast<const uint4*>(x + r * H)[c], xf);
            unpack8(reinterpret_cast<const uint4*>(dy + r * H)[c], df);
            const float rr = rstd[r];
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += df[e] * xf[e] * rr;
        }
        float4* o = reinterpret_cast<float4*>(dg_partial + static_cast<long long>(blockIdx.x) * H + c * 8);
        o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    }
}

// out[col] (+)= sum over parts of parts[p][col]. A block covers 32 columns. The rows form 32 chains, p modulo 32 (rows past the
// last round of four chains that are 8 apart go to the first of them), one warp each: what bounds this is the number of
// dependent loads in a row (eight warps with four chains each: 296 rows of 1000 and of 2048 columns, cold
// caches, 10.6 and 10.3 -> 5.5 us). Chains are added in fours, the eight sums in order.
constexpr int kReduceWarps = 32;
// Several sums of one width go out together, one to a row of blocks: in a chain of short kernels each launch costs what it takes.
struct ReduceJobs {
    cai_dg_sum job[CAI_DG_SUMS];
};
static __global__ void __launch_bounds__(kReduceWarps * 32)
reduce_parts_kernel(const __grid_constant__ ReduceJobs jobs, int H) {
    grid_dep_begin();
    const cai_dg_sum& job = jobs.job[blockIdx.y];
    const float* __restrict__ parts = job.partial;
    float* __restrict__ out = job.dg;
    const int nparts = job.parts, accumulate = job.accumulate;
    __shared__ float acc[kReduceWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = warp & 7, k = warp >> 3;
    const int col = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (col < H) {
        int p = w;
#pragma unroll 4
        for (; p + 24 < nparts; p += 32) s += parts[static_cast<long long>(p + 8 * k) * H + col];
        if (k == 0)
            for (; p < nparts; p += 8) s += parts[static_cast<long long>(p) * H + col];
    }
    acc[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && col < H) {
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) v += (acc[i][lane] + acc[i + 8][lane]) + (acc[i + 16][lane] + acc[i + 24][lane]);
        out[col] = accumulate ? out[col] + v : v;
    }
}

// Backward in ONE sweep for H <= 8192: a row is handled by R = ceil(H / 1024) warps that keep their slice of x and
// dy in registers (32 elements per lane), write dx and add the row's dy * x * rstd into per-lane column sums that
// they carry across all the rows they handle; at the end every warp leaves its sums in its own part of shared memory and the
// CTA adds them up (in a fixed order) to one partial row of the gain gradient. x and dy are read once (the
// two-kernel form above reads them twice), the old dx together with them. Two CTAs of eight warps share an SM.
// What bounds it is bytes in flight, and for few rows the combination of the sums: warps that took turns adding into one
// row, eight lanes to a bank, needed 3 us more.
// With an accumulated dx and cold caches, 16384 x 2048: 74.8 -> 58.5 us (4.6 TB/s), 3840 x 1000: 15.6 -> 12.8 us (before rows came ahead).
// Beside a product of another stream it runs on the SMs that one leaves free: none of its CTAs was seen to share an SM with a
// persistent product's, whatever the shared memory either asks for.
constexpr int kNormFusedThreads = 256;
constexpr int kNormStageBytes = 8 * kNormFusedCols * 2;   // a tensor's rows of one round: neighbours in memory, at most 8 x 1024 elements
// A CTA's rounds. Rows that did not come (a wait that ran out) are neither used nor followed by more: the phase of the barrier that they belong to is still
// open. The barrier behind the wait tells all threads alike (a word of shared memory read behind it cost 0.1 us a round).
struct NormRounds {
    struct Next { bool use, fetch; };
    long long first, step;         // first row of the round; rows that all CTAs take in one
    int rows;
    __host__ __device__ __forceinline__ NormRounds(int cta, int ctas, int groups, int rows_)
        : first(static_cast<long long>(cta) * groups), step(static_cast<long long>(ctas) * groups), rows(rows_) {}
    __host__ __device__ __forceinline__ bool more() const { return first < rows; }
    __host__ __device__ __forceinline__ Next behind_wait(bool came) const { return {came, came && first + step < rows}; }
};
// kStaged: a CTA's rows of the next round are on their way to shared memory, one bulk copy for each tensor, while this round's are worked on from
// registers. A warp that loads its own has nothing in flight while it computes and writes. us with the reduction, before /
// now, dx accumulated and written: 16384 x 2048 61.3 / 55.6 and 56.2 / 48.7 (4.8 and 4.1 TB/s), 5000 x 8192 77.6 / 72.5 and 69.9 / 62.4, 20000 x 256
// 19.6 / 16.6 and 18.1 / 15.8. Up to two rounds nothing is gained (3840 x 1000 12.8 / 12.9), and a warp loads its own rows.
template <bool kStaged>
static __global__ void __launch_bounds__(kNormFusedThreads, 2)
rmsnorm_bwd_fused_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ g,
                         const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ dy,
                         __nv_bfloat16* dx, float* __restrict__ dg_partial, int rows, int H, int dx_acc, int R, int* status) {
    extern __shared__ __align__(16) float sdg[];   // [warp][chunk * 8 + element][lane]: a warp's column sums, no two lanes on one bank
    __shared__ float part[8];
    __shared__ uint64_t landed;
    __shared__ volatile int abort_flag;
    uint8_t* const stage = reinterpret_cast<uint8_t*>(sdg + 8 * kNormFusedCols);   // x, dy, dx
    if constexpr (kStaged) {
        if (threadIdx.x == 0) {
            mbar_init(&landed, 1);
            abort_flag = 0;
            mbar_fence_init();
        }
        __syncthreads();
    }
    grid_dep_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = 8 / R;                 // rows a CTA works on at a time
    const int grp = warp / R, sub = warp - grp * R;
    const bool active = grp < groups;
    const int col0 = sub * kNormFusedCols;
    const uint4* gr = reinterpret_cast<const uint4*>(g);
    float acc[4][8];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[c][e] = 0.f;
    // one thread fetches the rows from `first` on
    auto fetch = [&](long long first) {
        const uint32_t bytes = static_cast<uint32_t>(rows - first < groups ? rows - first : groups) * static_cast<uint32_t>(H) * 2u;
        mbar_expect_tx(&landed, dx_acc ? 3 * bytes : 2 * bytes);
        bulk_load(stage, x + first * H, bytes, &landed);
        bulk_load(stage + kNormStageBytes, dy + first * H, bytes, &landed);
        if (dx_acc) bulk_load(stage + 2 * kNormStageBytes, dx + first * H, bytes, &landed);
    };
    NormRounds r(static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x), groups, rows);
    uint32_t round = 0;
    if (kStaged && threadIdx.x == 0 && r.more()) fetch(r.first);
    for (; r.more(); r.first += r.step, ++round) {
        const long long row = r.first + grp;
        const bool live = active && row < rows;
        uint4 xv[4], dv[4], old[4];
        float S = 0.f;
        const float rr = live ? rstd[row] : 0.f;      // asked for here: behind the sum it would be waited for
        const bool came = !kStaged || mbar_wait(&landed, round & 1, &abort_flag, status, CAI_DEV_TIMEOUT_TMA_FULL);
        if (live) {
            const uint4* xr = reinterpret_cast<const uint4*>(kStaged ? reinterpret_cast<const __nv_bfloat16*>(stage) + grp * H : x + row * H);
            const uint4* dyr = reinterpret_cast<const uint4*>(kStaged ? reinterpret_cast<const __nv_bfloat16*>(stage + kNormStageBytes) + grp * H : dy + row * H);
            const uint4* oldr = reinterpret_cast<const uint4*>(kStaged ? reinterpret_cast<const __nv_bfloat16*>(stage + 2 * kNormStageBytes) + grp * H : dx + row * H);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = col0 + (c * 32 + lane) * 8;
                if (col < H) {
                    xv[c] = xr[col >> 3];
                    dv[c] = dyr[col >> 3];
                    if (dx_acc) old[c] = oldr[col >> 3];
                }
            }
        }
        if (kStaged) {
            const NormRounds::Next next = r.behind_wait(__syncthreads_and(came));      // everybody has this round's rows in registers
            if (!next.use) {
                // the status word says so; copies under way are given time to land before the CTA's memory goes
                for (int i = 0; i < 32; ++i) __nanosleep(50000);
                break;
            }
            if (threadIdx.x == 0 && next.fetch) fetch(r.first + r.step);
        }
        if (live) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = col0 + (c * 32 + lane) * 8;
                if (col < H) {
                    float xf[8], df[8], gf[8];
                    unpack8(xv[c], xf);
                    unpack8(dv[c], df);
                    unpack8(gr[col >> 3], gf);
#pragma unroll
                    for (int e = 0; e < 8; ++e) S += df[e] * gf[e] * xf[e];
                }
            }
        }
        S = warp_sum(S);
        if (R > 1) {
            if (lane == 0) part[warp] = S;
            __syncthreads();
            if (active) {
                S = 0.f;
                for (int k = 0; k < R; ++k) S += part[grp * R + k];
            }
            __syncthreads();
        }
        if (live) {
            const float k3 = rr * rr * rr * S / H;
            uint4* dxr = reinterpret_cast<uint4*>(dx + row * H);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = col0 + (c * 32 + lane) * 8;
                if (col < H) {
                    float xf[8], df[8], gf[8], o[8];
                    unpack8(xv[c], xf);
                    unpack8(dv[c], df);
                    unpack8(gr[col >> 3], gf);
                    if (dx_acc) unpack8(old[c], o);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float v = rr * df[e] * gf[e] - k3 * xf[e];
                        o[e] = dx_acc ? o[e] + v : v;
                        acc[c][e] += df[e] * xf[e] * rr;
                    }
                    dxr[col >> 3] = pack8(o);
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int e = 0; e < 8; ++e) sdg[(warp * 32 + c * 8 + e) * 32 + lane] = acc[c][e];
    __syncthreads();
    // column of slice `sl`: chunk, lane and element from its place; row groups in order, so the result does not depend on timing
    for (int i = threadIdx.x; i < R * kNormFusedCols; i += kNormFusedThreads) {
        const int sl = i / kNormFusedCols, in = i - sl * kNormFusedCols;    // in = (chunk * 8 + element) * 32 + lane
        const int col = sl * kNormFusedCols + ((in >> 8) * 32 + (in & 31)) * 8 + ((in >> 5) & 7);
        if (col < H) {
            float v = 0.f;
            for (int w = 0; w < groups; ++w) v += sdg[(w * R + sl) * kNormFusedCols + in];
            dg_partial[static_cast<long long>(blockIdx.x) * H + col] = v;
        }
    }
}

static inline int launch_reduce_parts(const cai_dg_sum* sums, int n, int H, cudaStream_t st) {
    ReduceJobs jobs = {};
    for (int i = 0; i < n; ++i) jobs.job[i] = sums[i];
    launch_early(reduce_parts_kernel, dim3((H + 31) / 32, n), kReduceWarps * 32, 0, st, jobs, H);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// The one-sweep form without the reduction of its `grid` partial rows.
static inline int launch_rmsnorm_sweep(const void* x, const void* g, const float* rstd, const void* dy, void* dx, float* partial, int grid, int rows, int H,
                                       int dx_accumulate, cudaStream_t st) {
    const int Rf = rmsnorm_fused_row_warps(H), groups = 8 / Rf;
    const long long want = (static_cast<long long>(rows) + groups - 1) / groups;
    constexpr size_t smem = 8 * kNormFusedCols * sizeof(float), smem_staged = smem + 3 * kNormStageBytes;
    const bool staged = want > 2LL * grid;                 // three rounds and more
    if (staged) {
        static bool configured[64] = {};
        const int dev = current_device();
        if (!configured[dev & 63]) {
            if (cudaFuncSetAttribute(rmsnorm_bwd_fused_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_staged)) != cudaSuccess) return 1;
            configured[dev & 63] = true;
        }
    }
    launch_early(staged ? rmsnorm_bwd_fused_kernel<true> : rmsnorm_bwd_fused_kernel<false>, grid, kNormFusedThreads, staged ? smem_staged : smem, st,
                 static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(g), rstd, static_cast<const __nv_bfloat16*>(dy),
                 static_cast<__nv_bfloat16*>(dx), partial, rows, H, dx_accumulate, Rf, status_words(current_device()));
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// Host side of RMSNorm backward, shared by the entry points: `scratch` holds at most `parts_cap`
// rows of H floats. Returns a cudaError_t-style 0 / non-zero.
static inline int launch_rmsnorm_bwd(const void* x, const void* g, const float* rstd, const void* dy, void* dx, float* dg,
                                     float* scratch, int parts_cap, int sms, int rows, int H, int dx_accumulate,
                                     int dg_accumulate, cudaStream_t st) {
    if (H <= kNormFusedMaxH && (H & 7) == 0 && parts_cap >= 1) {
        // one sweep: dx and the partial gain gradients from the same read of x and dy
        const int grid = rmsnorm_fused_parts(rows, H, parts_cap, sms);
        if (launch_rmsnorm_sweep(x, g, rstd, dy, dx, scratch, grid, rows, H, dx_accumulate, st)) return 1;
        const cai_dg_sum sum = {scratch, dg, grid, dg_accumulate};
        return launch_reduce_parts(&sum, 1, H, st);
    }
    const int R = (H + kNormWarpCols - 1) / kNormWarpCols;
    const int groups = 8 / R;
    const long long want = (static_cast<long long>(rows) + groups - 1) / groups;
    const int grid = static_cast<int>(want < sms * 8LL ? want : sms * 8LL);
    int parts = rows < parts_cap ? rows : parts_cap;
    const int rows_per_part = (rows + parts - 1) / parts;
    parts = (rows + rows_per_part - 1) / rows_per_part;
    launch_early(rmsnorm_bwd_dg_kernel, parts, 256, 0, st, static_cast<const __nv_bfloat16*>(x), rstd,
                 static_cast<const __nv_bfloat16*>(dy), scratch, rows, H, rows_per_part);
    const cai_dg_sum sum = {scratch, dg, parts, dg_accumulate};
    if (launch_reduce_parts(&sum, 1, H, st)) return 1;
    // dx last: callers may pass dx == dy (in place), and the gain gradient needs the unmodified dy
    launch_early(rmsnorm_bwd_dx_kernel, grid, kNormThreads, 0, st, static_cast<const __nv_bfloat16*>(x),
                 static_cast<const __nv_bfloat16*>(g), rstd, static_cast<const __nv_bfloat16*>(dy), static_cast<__nv_bfloat16*>(dx), rows,
                 H, dx_accumulate, R);
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

}  // namespace cai
