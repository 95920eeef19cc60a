// backend_calibrated.cc - a pricing backend whose costs are fitted to measurements on B200s.
//
// The analytic backend keeps the reference's model (FLOPs over the datasheet peak, bytes over the link figure:
// src/backend_cpu.c:28-49), which is what its published predictions are made of. This backend prices the same
// executable plans with what the kernels of this repository were measured to do, so that a configuration can be
// judged without a GPU: the replayer (runtime_sim.cc) walks the op table over the six stream clocks as before, and
// additionally keeps the step from being shorter than the GPU-filling work of all streams together (two kernels that
// each fill the GPU do not speed each other up by sitting on different streams).
//
// Model per kernel (constants: `Calibration`, overridable from a key = value file; sources in the comments there):
//   GEMM            launch + waves * (tile overhead + tile FLOPs / per-SM rate): tiles of 256 x 256 or 256 x 128 on 74 pairs of SMs, or
//                   a slice of K of one, as the kernel's own rule has it; a lower rate for transposed-A products (weight
//                   gradients). Products fused with a collective, SwiGLU's backward epilogue and e4m3: 128 x 256 (or 128 x
//                   128) tiles on 148 SMs with constants of their own
//   attention       per-CTA critical path: steps = max(all steps / SMs, longest CTA) * time per 128 x 128 step
//   pointwise       per-kernel fixed cost + operand bytes * per-kernel microseconds per MB
//   fused TP ops    launch + max(GEMM on the SMs left beside the copy CTAs, wire bytes / measured rate under all-to-all
//                   load for the group size) (+ the own-row tail of the reduce-scatter)
//   NCCL, p2p       latency + bytes / rate
//   joined records  what an untraced step launches instead (csrc/runtime/launches.h): two products as one schedule of both one's tiles, a projection with its
//                   SwiGLU as one product, a rotation behind an attention backward and results that nobody reads as nothing, the last sums of
//                   RMSNorm backward once for all that wait. Timelines are of single records, as traced steps run them
// Fixed costs are those of an untraced step, where plain kernels are launched while their predecessor finishes. The per-op events of a
// traced step keep an op from starting early: each takes some 5 us more there (before records went out together, 52 ops of a tiny step 593 us by their
// events, 331 us without; 137 of a small one 4182 and 3531).
// Needs a version-2 plan (kernel records and shapes); version-1 plans fall back to the analytic cost.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <sstream>

#include "../runtime/launches.h"
#include "backend.h"

namespace cai {
namespace {

struct PointCost {
    double fixed_us;
    double us_per_mb;
};

struct Calibration {
    int sms = 148;
    // Plain GEMM, fitted to the per-op CUDA-event times inside steps of six models on one GPU (the headline config in launches of
    // 16384 and of 4096 tokens, two of its layers' tensor-parallel shards as models of their own, two 8B-class layers, a
    // small ragged model; 90 shapes, median error 4 %), less what an op starts early: [0] A not transposed, [1] A transposed
    // (weight-gradient form). The fixed costs here and below are since set by twelve models, less what a traced op takes more; their untraced steps,
    // predicted / measured on one B200, ms: 59.8 / 61.5, 18.2 / 18.2, 27.5 / 28.6, 47.3 / 48.0, 17.1 / 17.4, 5.19 / 4.93, 4.94 / 5.06, 3.52 / 3.71,
    // 3.25 / 3.16, 3.06 / 3.08, 1.83 / 1.92, 0.248 / 0.251
    double gemm_launch_us = 4.0;
    double gemm_tile_us[2] = {1.9, 0.2};
    double gemm_sm_flops[2] = {10.7e12, 9.4e12};
    int joins = 1;                  // 0: every record by itself, as kernels before there were joined forms ran them
    int gemm_pairs = 1;             // 0: plain products run one CTA per 128-row tile, as the fused ones do
    // One-CTA GEMM (fused with a collective): the headline config's shapes on one GPU, fit error <= 13 %
    double fused_gemm_tile_us = 0.5;
    double fused_gemm_sm_flops = 7.9e12;
    // fp8 block-scaled GEMM against the one-CTA bf16 one: inside steps of two models, 1.5 (hidden 1024) and 2.2 (hidden 4096)
    double fp8_speedup = 1.9;
    // attention, microseconds per 128 x 128 step of one CTA (the same six models)
    double attn_fwd_step_us = 1.59, attn_fwd_fixed_us = 7.0;
    double attn_dkdv_step_us = 2.53, attn_dq_step_us = 2.00, attn_bwd_fixed_us = 11.8;
    double dg_sums_us = 3.0;        // the last sums of RMSNorm backward, which a norm by itself launches too
    // fused tensor-parallel kernels: bytes a GPU moves per second while every member pulls and pushes at once
    // (steady-state chains on 2 / 4 / 8 GPUs), copy CTAs of the all-gather form, tail of the reduce-scatter form
    double link_rate[4] = {0.60e12, 0.60e12, 0.45e12, 0.35e12};  // group size 1-2, 2, 4, 8
    int ag_copy_ctas = 16;
    double rs_tail_us = 35.0;
    double fused_launch_us = 15.0;
    double fused_min_share = 0.6;
    // NCCL collectives and p2p next to compute
    double nccl_latency_us = 20.0;
    double nccl_rate = 0.60e12;   // bytes per GPU and second of ring collectives of 17-120 MB (NCCL arms of the chains)
    // pointwise kernels (the same six models; worst errors 6-14 %, the embedding's backward apart, whose time goes with how
    // often a token repeats)
    PointCost point_default = {3.3, 0.20};
    PointCost rmsnorm_fwd = {1.7, 0.181}, rmsnorm_bwd = {6.0, 0.305}, rope = {1.1, 0.332}, swiglu = {0.6, 0.170},
              adamw = {0.0, 0.2456}, cross_entropy = {9.5, 0.470}, embed = {6.0, 0.25};
};

bool set_key(Calibration* c, const std::string& k, double v) {
    struct Entry { const char* name; double* dst; };
    Entry table[] = {
        {"gemm_launch_us", &c->gemm_launch_us}, {"gemm_tile_us", &c->gemm_tile_us[0]}, {"gemm_tile_us_ta", &c->gemm_tile_us[1]},
        {"gemm_sm_flops", &c->gemm_sm_flops[0]}, {"gemm_sm_flops_ta", &c->gemm_sm_flops[1]}, {"fp8_speedup", &c->fp8_speedup},
        {"fused_gemm_tile_us", &c->fused_gemm_tile_us}, {"fused_gemm_sm_flops", &c->fused_gemm_sm_flops},
        {"attn_fwd_step_us", &c->attn_fwd_step_us}, {"attn_fwd_fixed_us", &c->attn_fwd_fixed_us},
        {"attn_dkdv_step_us", &c->attn_dkdv_step_us}, {"attn_dq_step_us", &c->attn_dq_step_us},
        {"attn_bwd_fixed_us", &c->attn_bwd_fixed_us}, {"link_rate_2", &c->link_rate[1]}, {"link_rate_4", &c->link_rate[2]},
        {"link_rate_8", &c->link_rate[3]}, {"rs_tail_us", &c->rs_tail_us}, {"fused_launch_us", &c->fused_launch_us},
        {"dg_sums_us", &c->dg_sums_us}, {"nccl_latency_us", &c->nccl_latency_us}, {"nccl_rate", &c->nccl_rate}, {"fused_min_share", &c->fused_min_share},
    };
    for (const Entry& e : table)
        if (k == e.name) {
            *e.dst = v;
            return true;
        }
    struct PEntry { const char* name; PointCost* dst; };
    PEntry points[] = {{"pointwise", &c->point_default}, {"rmsnorm_fwd", &c->rmsnorm_fwd}, {"rmsnorm_bwd", &c->rmsnorm_bwd},
                       {"rope", &c->rope}, {"swiglu", &c->swiglu}, {"adamw", &c->adamw}, {"cross_entropy", &c->cross_entropy},
                       {"embed", &c->embed}};
    for (const PEntry& e : points) {   // <kernel>_fixed_us, <kernel>_us_per_mb
        const std::string n = e.name;
        if (k == n + "_fixed_us") { e.dst->fixed_us = v; return true; }
        if (k == n + "_us_per_mb") { e.dst->us_per_mb = v; return true; }
    }
    if (k == "sms") { c->sms = static_cast<int>(v); return true; }
    if (k == "joins") { c->joins = v != 0.0; return true; }
    if (k == "gemm_pairs") { c->gemm_pairs = v != 0.0; return true; }
    if (k == "ag_copy_ctas") { c->ag_copy_ctas = static_cast<int>(v); return true; }
    return false;
}

struct CalibratedImpl {
    Calibration c;
    std::vector<ExecOp> exec;
    std::vector<TensorDesc> tensors;
    uint32_t capacity_x100 = 200;
    // How a record goes out in an untraced step: the (first) record of a launch with the one behind it, or none (it goes out with the one before, or not at all);
    // sums that go out behind a sweep.
    struct Joined {
        enum How : uint8_t { kRecord, kTwoProducts, kSwiglu, kRotated, kNormSweep, kNothing } how = kRecord;
        uint32_t next = 0;
        int sums = 0;
    };
    std::vector<Joined> joined;
    bool join = false;
};

// One CTA per tile of 128 rows.
double one_cta_gemm_seconds(const Calibration& c, double tile_us, double sm_flops, double M, double N, double K, int sms, double* share) {
    const double bn = (static_cast<long long>(N) % 256 == 0) ? 256.0 : 128.0;
    const double tiles = std::ceil(M / 128.0) * std::ceil(N / bn);
    const double waves = std::max(1.0, std::ceil(tiles / sms));
    if (share) *share = std::min(1.0, tiles / (waves * c.sms));
    return (c.gemm_launch_us + waves * (tile_us + 2.0 * 128.0 * bn * K / sm_flops * 1e6)) * 1e-6;
}

double fused_gemm_seconds(const Calibration& c, double M, double N, double K, int sms, double* share) {
    return one_cta_gemm_seconds(c, c.fused_gemm_tile_us, c.fused_gemm_sm_flops, M, N, K, sms, share);
}

// A plain product: pairs of SMs, a tile of 256 rows each. The form is chosen as the kernel chooses it (cycles per 128 k-elements and per
// tile, see csrc/kernels/gemm_pair.cu); a 128-wide tile takes 0.74 of a 256-wide one's time.
double gemm_seconds(const Calibration& c, double M, double N, double K, bool ta, int sms, double* share, double groups = 1.0) {
    const int cls = ta ? 1 : 0;
    if (!c.gemm_pairs) return one_cta_gemm_seconds(c, c.gemm_tile_us[cls], c.gemm_sm_flops[cls], M, N, K, sms, share);
    const double pairs = std::max(1.0, std::floor(sms / 2.0)), ks = std::ceil(K / 128.0), tm = std::ceil(M / 256.0);
    const double t256 = tm * std::ceil(N / 256.0) * groups, t128 = tm * std::ceil(N / 128.0) * groups;
    const double w256 = std::max(1.0, std::ceil(t256 / pairs)), w128 = std::max(1.0, std::ceil(t128 / pairs));
    const double wide = w256 * (ks * 1150.0 + 2500.0), narrow = w128 * (ks * 850.0 + 1500.0);
    const double two = ks >= 2 && t128 <= 33 ? std::ceil(ks / 2.0) * 850.0 + 4500.0 : 1e30;
    const double four = ks >= 4 && t128 <= 15 ? std::ceil(ks / 4.0) * 850.0 + 4500.0 : 1e30;
    const double full = 2.0 * 256.0 * 256.0 * K / (2.0 * c.gemm_sm_flops[cls]) * 1e6;   // a 256-wide tile on a pair, microseconds
    double waves = w256, tiles = t256, work = full;
    if (four < two && four < wide && four < narrow) {
        waves = 1.0; tiles = 4.0 * t128; work = 0.74 / 4.0 * full;
    } else if (two < wide && two < narrow) {
        waves = 1.0; tiles = 2.0 * t128; work = 0.74 / 2.0 * full;
    } else if (narrow < wide) {
        waves = w128; tiles = t128; work = 0.74 * full;
    }
    if (share) *share = std::min(1.0, tiles / (waves * (c.sms / 2.0)));
    return (c.gemm_launch_us + waves * (c.gemm_tile_us[cls] + work)) * 1e-6;
}

// Two plain products that can go out together: one launch of both one's tiles, or slices of tiles that all run at once.
double two_products_seconds(const Calibration& c, const ExecOp& x, const ExecOp& y, int sms, double* share) {
    const ExecOp* o[2] = {&x, &y};
    PairTwoForm f;
    double s[2], w[2], t[2];
    if (!c.gemm_pairs || !pair_two_form({x.i[0], x.i[1], x.i[2], epilogue(x)}, {y.i[0], y.i[1], y.i[2], epilogue(y)}, &f)) {
        for (int k = 0; k < 2; ++k) s[k] = gemm_seconds(c, o[k]->i[0], o[k]->i[1], o[k]->i[2], o[k]->flags & 1, sms, &w[k]);
        if (share) *share = (s[0] * w[0] + s[1] * w[1]) / (s[0] + s[1]);
        return s[0] + s[1];
    }
    long long n[2];
    for (int k = 0; k < 2; ++k) {
        const int cls = o[k]->flags & 1;
        n[k] = pair_tile_count(o[k]->i[0], o[k]->i[1], f.tile_cols);
        t[k] = c.gemm_tile_us[cls] + (f.tile_cols == 256 ? 1.0 : 0.74) / f.slices[k] * 2.0 * 256.0 * 256.0 * o[k]->i[2] / (2.0 * c.gemm_sm_flops[cls]) * 1e6;
    }
    const long long pairs = std::max(1, sms / 2);
    double us = std::max(t[0], t[1]);                       // split: every slice runs at once
    if (f.slices[0] == 1 && f.slices[1] == 1) {
        int heavier, more;
        us = pair_two_schedule(n[f.first], t[f.first], n[1 - f.first], t[1 - f.first], std::min(pairs, n[0] + n[1]), &heavier, &more);
    }
    if (share) *share = std::min(1.0, (n[0] * t[0] * f.slices[0] + n[1] * t[1] * f.slices[1]) / (us * (c.sms / 2.0)));
    return (c.gemm_launch_us + us) * 1e-6;
}

double operand_mb(const CalibratedImpl& im, const ExecOp& x) {
    double b = 0.0;
    for (int t : x.t)
        if (t >= 0 && static_cast<size_t>(t) < im.tensors.size()) b += static_cast<double>(im.tensors[t].nbytes);
    return b / 1e6;
}

double link_rate(const Calibration& c, uint32_t n) { return c.link_rate[n <= 2 ? 1 : n <= 4 ? 2 : 3]; }

constexpr double kBothParts = 1.8;       // steps of dK / dV that both parts' steps on an SM come to, one of each (the steps' times above)

// Seconds and the share of the GPU's SMs the op keeps busy while it runs.
double price(const CalibratedImpl& im, const Topology& topo, const Op& op, const CommGroup* g, double* share) {
    const Calibration& c = im.c;
    *share = 1.0;
    if (!op.exec || op.exec > im.exec.size()) {
        *share = op_is_compute(op.kind) ? 1.0 : 0.0;
        return analytic_op_seconds(topo, op, g);
    }
    const ExecOp& x = im.exec[op.exec - 1];
    const uint32_t n = g ? g->size : 1;
    const CalibratedImpl::Joined joined = im.join ? im.joined[op.exec - 1] : CalibratedImpl::Joined{};
    if (joined.how == CalibratedImpl::Joined::kNothing) {
        *share = 0.0;
        return 0.0;
    }
    if (joined.how == CalibratedImpl::Joined::kTwoProducts) return two_products_seconds(c, x, im.exec[joined.next], c.sms, share);
    auto point = [&](const PointCost& pc) { return (pc.fixed_us + operand_mb(im, x) * pc.us_per_mb) * 1e-6; };
    switch (x.kernel) {
    case K_GEMM: {
        double M = x.i[0], N = x.i[1], K = x.i[2];
        if (x.flags & 0x100) {
            // grouped expert GEMM: one launch over all local experts' slabs (op.flops counts every slab row); tiles past a
            // slab's token count are skipped, and with balanced routing a slab is filled to 1 / capacity factor
            const double experts = std::max(1.0, std::round(static_cast<double>(op.flops) / (2.0 * M * N * K)));
            const double live = std::min(1.0, 100.0 / std::max(100u, im.capacity_x100));
            if (x.i[4] == 2050) K *= live;   // weight-gradient form: the ragged dimension is K
            else M *= live;
            if (x.i[4] == 2050)
                return c.gemm_pairs ? gemm_seconds(c, M, N, K, x.flags & 1, c.sms, share, experts)
                                    : experts * gemm_seconds(c, M, N, K, x.flags & 1, c.sms, share);
            M *= experts;
        }
        if (((x.flags >> 4) & 0xF) == 5 && c.gemm_pairs) return fused_gemm_seconds(c, M, N, K, c.sms, share);   // CAI_EPI_SWIGLU_BWD
        return gemm_seconds(c, M, N, K, x.flags & 1, c.sms, share);
    }
    case K_GEMM_FP8:
        return fused_gemm_seconds(c, x.i[0], x.i[1], x.i[2], c.sms, share) / c.fp8_speedup;
    case K_AG_GEMM: case K_GEMM_RS: {
        const bool ag = x.kernel != K_GEMM_RS;
        const double compute = fused_gemm_seconds(c, x.i[0], x.i[1], x.i[2], ag ? c.sms - c.ag_copy_ctas : c.sms, nullptr);
        const double wire = n > 1 ? (n - 1.0) / n * static_cast<double>(op.bytes) / link_rate(c, n) : 0.0;
        const double tail = (x.kernel == K_GEMM_RS && n > 1) ? c.rs_tail_us * 1e-6 : 0.0;
        const double dur = c.fused_launch_us * 1e-6 + std::max(compute, wire) + tail;
        // a transfer-bound call leaves issue slots and memory bandwidth to kernels of other streams while it waits
        *share = compute >= wire ? 1.0 : std::max(c.fused_min_share, compute / wire);
        return dur;
    }
    case K_ATTN_FWD: case K_ATTN_BWD: {
        const double B = x.i[0], S = x.i[1], nh = x.i[2], nkv = std::max(1, x.i[3]);
        const double nq = S / 128.0, tri = nq * (nq + 1.0) / 2.0, rep = nh / nkv;
        if (x.kernel == K_ATTN_FWD) {
            const double steps = std::max(B * nh * tri / c.sms, nq);
            *share = std::min(1.0, B * nh * nq / c.sms);
            return (c.attn_fwd_fixed_us + steps * c.attn_fwd_step_us) * 1e-6;
        }
        // parts (flags): bit 0 delta, bit 1 dK / dV, bit 2 dQ; 0 means all three
        const int parts = (x.flags & 7) ? (x.flags & 7) : 7;
        double t = c.attn_bwd_fixed_us;
        // dK / dV: one CTA per (kv tile, kv group) sweeping the group's heads, or per query head when that grid fits the SMs
        const bool split = rep > 1 && B * nkv * nq < c.sms && B * nh * nq <= c.sms;
        const double steps = B * nh * tri / c.sms, longest = (split ? 1.0 : rep) * nq;
        if ((parts & 6) == 6 && longest > kBothParts * steps) t += longest * c.attn_dkdv_step_us;      // one launch: dQ's CTAs run beside the longest
        else {
            if (parts & 2) t += std::max(steps, (parts & 4) ? 0.0 : longest) * c.attn_dkdv_step_us;
            if (parts & 4) t += std::max(steps, (parts & 2) ? 0.0 : nq) * c.attn_dq_step_us;
        }
        *share = std::min(1.0, B * nh * nq / c.sms);
        return t * 1e-6;
    }
    case K_RMSNORM_FWD: return point(c.rmsnorm_fwd);
    case K_RMSNORM_BWD:
        if (joined.how == CalibratedImpl::Joined::kNormSweep) return std::max(0.0, point(c.rmsnorm_bwd) - c.dg_sums_us * 1e-6) + joined.sums * c.dg_sums_us * 1e-6;
        return point(c.rmsnorm_bwd);
    case K_ROPE: return point(c.rope);
    case K_SWIGLU_FWD: case K_SWIGLU_BWD: return point(c.swiglu);
    case K_ADAMW: return point(c.adamw);
    case K_CROSS_ENTROPY: case K_CROSS_ENTROPY_TP: return point(c.cross_entropy);
    case K_EMBED_FWD: case K_EMBED_BWD: return point(c.embed);
    case K_FSDP_AG_GEMM: {
        // ZeRO-3 parameter gather of one group (op.bytes = what crosses the links); flag 1: the copy CTAs ride in the
        // first GEMM that reads the group, which measured slower than the transfer alone (482 us against 406 us of
        // all-gather + GEMM at 2 GPUs for a 50 MB group), priced here as twice the transfer
        const double wire = static_cast<double>(op.bytes) / link_rate(c, n);
        *share = 0.2;
        return c.fused_launch_us * 1e-6 + ((x.flags & 1) ? 2.0 : 1.0) * wire;
    }
    case K_RS_ADAMW: {
        // reduce-scatter + AdamW (+ parameter all-gather) over the data-parallel group. op.flops = 18 per element of
        // the owned slice: the slice's optimizer traffic, and (n - 1) x 6 bytes per owned element over the links
        // (fp32 gradients in, bf16 parameters out). 1.72 ms for 256 Mi parameters on 2 GPUs.
        const double owned = static_cast<double>(op.flops) / 18.0;
        const double opt = (c.adamw.fixed_us + owned * 18.0 / 1e6 * c.adamw.us_per_mb) * 1e-6;
        const double wire = n > 1 ? (n - 1.0) * owned * 6.0 / link_rate(c, n) : 0.0;
        *share = 0.45;  // launched on a slice of the SMs beside the backward
        return c.fused_launch_us * 1e-6 + std::max(opt, wire) + 0.5 * std::min(opt, wire);
    }
    case K_NCCL_ALL_REDUCE: case K_NCCL_REDUCE_SCATTER: case K_NCCL_ALL_GATHER: case K_NCCL_ALL_TO_ALL:
    case K_NCCL_SEND: case K_NCCL_RECV: {
        *share = 0.15;  // NCCL's own CTAs
        // op.bytes: the whole tensor for an all-reduce, this rank's shard for the others
        double wire = static_cast<double>(op.bytes);
        if (x.kernel == K_NCCL_ALL_REDUCE) wire *= n > 1 ? 2.0 * (n - 1.0) / n : 0.0;
        else if (x.kernel != K_NCCL_SEND && x.kernel != K_NCCL_RECV) wire *= n > 1 ? n - 1.0 : 0.0;
        return c.nccl_latency_us * 1e-6 + wire / c.nccl_rate;
    }
    case K_MOE_DISPATCH_GEMM: case K_MOE_GEMM_COMBINE: {
        const double wire = n > 1 ? (n - 1.0) / n * static_cast<double>(op.bytes) / link_rate(c, n) : 0.0;
        return c.fused_launch_us * 1e-6 + std::max(point(c.point_default), wire);
    }
    default:
        *share = 0.5;
        return point(c.point_default);
    }
}

double calibrated_op_seconds(Backend* be, const Topology& topo, const Op& op, const CommGroup* g) {
    double share;
    return price(*static_cast<CalibratedImpl*>(be->impl), topo, op, g, &share);
}

double calibrated_sm_share(Backend* be, const Topology& topo, const Op& op, const CommGroup* g) {
    double share = 0.0;
    price(*static_cast<CalibratedImpl*>(be->impl), topo, op, g, &share);
    return share;
}

int calibrated_load_plan(Backend* be, const Plan& plan, const std::string&, uint32_t, uint32_t) {
    auto* im = static_cast<CalibratedImpl*>(be->impl);
    im->exec = plan.exec;
    im->tensors = plan.tensors;
    im->capacity_x100 = plan.train.moe_capacity_factor_x100 ? plan.train.moe_capacity_factor_x100 : 200;
    im->joined.assign(plan.exec.size(), {});
    if (plan.exec.empty()) return OK;
    using Joined = CalibratedImpl::Joined;
    const std::vector<uint8_t> joins = find_joins(plan);
    LaunchWalk walk(plan, joins, true, true, im->c.sms);
    for (Joined& j : im->joined) j.how = Joined::kNothing;
    uint32_t sweep = 0;
    for (Launch l; walk.next(&l);) {
        if (l.what == Launch::kEvent) continue;
        if (l.what == Launch::kNormSums) {
            ++im->joined[sweep].sums;
            continue;
        }
        const uint32_t at = plan.ops[l.op].exec - 1;
        Joined& j = im->joined[at];
        j.how = l.what == Launch::kTwoProducts ? Joined::kTwoProducts : l.what == Launch::kSwiglu ? Joined::kSwiglu : l.what == Launch::kRotated ? Joined::kRotated
                : l.what == Launch::kNormSweep ? Joined::kNormSweep : Joined::kRecord;
        if (l.what == Launch::kTwoProducts) j.next = plan.ops[l.op + 1].exec - 1;
        if (l.what == Launch::kNormSweep) sweep = at;
    }
    return OK;
}

void calibrated_price_launches(Backend* be, bool on) {
    auto* im = static_cast<CalibratedImpl*>(be->impl);
    im->join = on && im->c.joins && im->joined.size() == im->exec.size();
}

void calibrated_destroy(Backend* be) {
    delete static_cast<CalibratedImpl*>(be->impl);
    delete be;
}

}  // namespace

Backend* backend_calibrated_create(const char* calibration_path, std::string* why) {
    auto im = new CalibratedImpl();
    if (calibration_path && *calibration_path) {
        std::ifstream f(calibration_path);
        if (!f) {
            if (why) *why = std::string("cannot read calibration file ") + calibration_path;
            delete im;
            return nullptr;
        }
        std::string line;
        int lineno = 0;
        while (std::getline(f, line)) {
            ++lineno;
            const size_t hash = line.find('#');
            if (hash != std::string::npos) line.resize(hash);
            const size_t eq = line.find('=');
            if (eq == std::string::npos) continue;
            auto trim = [](std::string s) {
                const size_t a = s.find_first_not_of(" \t\r"), b = s.find_last_not_of(" \t\r");
                return a == std::string::npos ? std::string() : s.substr(a, b - a + 1);
            };
            const std::string k = trim(line.substr(0, eq)), v = trim(line.substr(eq + 1));
            char* end = nullptr;
            const double val = std::strtod(v.c_str(), &end);
            if (k.empty() || end == v.c_str() || !set_key(&im->c, k, val)) {
                if (why) {
                    std::ostringstream o;
                    o << calibration_path << ":" << lineno << ": unknown key or bad value '" << k << "'";
                    *why = o.str();
                }
                delete im;
                return nullptr;
            }
        }
    }
    auto be = new Backend();
    be->name = "calibrated";
    be->impl = im;
    be->op_seconds = calibrated_op_seconds;
    be->op_sm_share = calibrated_sm_share;
    be->load_plan = calibrated_load_plan;
    be->price_launches = calibrated_price_launches;
    be->run_step = nullptr;
    be->snapshot = nullptr;
    be->restore = nullptr;
    be->sync = nullptr;
    be->destroy = calibrated_destroy;
    return be;
}

}  // namespace cai
