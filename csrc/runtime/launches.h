// launches.h - what a replay of a plan launches, in order.
//
// The plan names every operation. A replay joins neighbours on one stream, leaves out what nobody reads and lets the last sums of
// RMSNorm backward wait for each other. Which ones follows from the plan's records and the bytes that they name, so it is decided here, without a
// GPU: the executor carries the list out, the calibrated backend prices it, and cai_plan_launches shows it.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../kernels/cai_kernels.h"
#include "../kernels/norm_form.h"
#include "../kernels/pair_form.h"
#include "../plan/plan.h"

namespace cai {

// How a record goes out: by itself; together with the one behind it (two products in one launch, a projection with the SwiGLU of its result, an attention
// backward with the rotation of its result); not at all.
enum Join : uint8_t { kAlone, kPairOfProducts, kWithSwiglu, kWithRotation, kUnread };

struct Bytes {
    uint64_t lo = 0, hi = 0;
    bool meets(const Bytes& o) const { return lo < o.hi && o.lo < hi; }
};

inline bool has_tensor(const Plan& p, int t) { return t >= 0 && static_cast<size_t>(t) < p.tensors.size(); }
inline Bytes tensor_bytes(const Plan& p, int t) {
    return has_tensor(p, t) ? Bytes{p.tensors[t].offset, p.tensors[t].offset + p.tensors[t].nbytes} : Bytes{};
}
inline long long pitch(const Plan& p, int t) { return p.shapes[static_cast<size_t>(t) * 4 + 2]; }
// The bytes of `rows` rows of `cols` elements, from the start of tensor t.
inline Bytes rows_of(const Plan& p, int t, long long rows, long long cols, int bytes) {
    if (!has_tensor(p, t) || rows <= 0) return {};
    return {p.tensors[t].offset, p.tensors[t].offset + static_cast<uint64_t>(((rows - 1) * pitch(p, t) + cols) * bytes)};
}

// A plain product: not of several groups, not ragged.
inline bool plain_product(const ExecOp& x) { return x.kernel == K_GEMM && !(x.flags & 0x100) && x.t[4] < 0; }
inline int epilogue(const ExecOp& x) { return (x.flags >> 4) & 0xF; }
inline Bytes operand_a(const Plan& p, const ExecOp& x) { return x.flags & 1 ? rows_of(p, x.t[0], x.i[2], x.i[0], 2) : rows_of(p, x.t[0], x.i[0], x.i[2], 2); }
inline Bytes operand_b(const Plan& p, const ExecOp& x) { return x.flags & 2 ? rows_of(p, x.t[1], x.i[2], x.i[1], 2) : rows_of(p, x.t[1], x.i[1], x.i[2], 2); }
inline Bytes result_c(const Plan& p, const ExecOp& x) {
    return rows_of(p, x.t[2], x.i[0], x.i[1], epilogue(x) == CAI_EPI_F32 || epilogue(x) == CAI_EPI_F32_ACCUM ? 4 : 2);
}

inline bool neighbours(const Op& a, const Op& b) {
    auto event = [](const Op& o) { return o.kind == OP_EVENT_RECORD || o.kind == OP_EVENT_WAIT; };
    return a.exec && b.exec && a.stream_id == b.stream_id && !event(a) && !event(b);
}

// Whether two records next to each other are plain products of which neither touches what the other writes: a layer's input gradient and weight
// gradient, which the plan puts side by side.
inline bool independent_products(const Plan& p, const ExecOp& x, const ExecOp& y) {
    const ExecOp* o[2] = {&x, &y};
    Bytes reads[2][3], writes[2];
    for (int k = 0; k < 2; ++k) {
        if (!plain_product(*o[k]) || epilogue(*o[k]) > CAI_EPI_BF16_RESIDUAL) return false;
        for (int t = 0; t < 3; ++t)
            if (!has_tensor(p, o[k]->t[t])) return false;
        reads[k][0] = operand_a(p, *o[k]);
        reads[k][1] = operand_b(p, *o[k]);
        if (epilogue(*o[k]) == CAI_EPI_BF16_RESIDUAL) reads[k][2] = rows_of(p, o[k]->t[3], o[k]->i[0], o[k]->i[1], 2);
        writes[k] = result_c(p, *o[k]);
    }
    if (writes[0].meets(writes[1])) return false;
    for (int k = 0; k < 2; ++k)
        for (const Bytes& r : reads[k])
            if (writes[1 - k].meets(r)) return false;
    return true;
}

// Whether two records next to each other are a gate / up projection and the SwiGLU of its result, of a width that the plan compiler leaves
// apart (F no multiple of 128), and one product with SwiGLU in its epilogue is the faster way. Tiles of the activation are written while others still read the
// operands: it must not lie over them, as it may where the two go out one behind the other.
inline bool projection_with_swiglu(const Plan& p, const ExecOp& x, const ExecOp& y) {
    if (!p.train.fuse_swiglu || !plain_product(x) || y.kernel != K_SWIGLU_FWD) return false;
    if (!has_tensor(p, x.t[0]) || !has_tensor(p, x.t[1]) || !has_tensor(p, x.t[2]) || !has_tensor(p, y.t[0]) || !has_tensor(p, y.t[1])) return false;
    if (epilogue(x) != CAI_EPI_BF16 || (x.flags & 3) || x.f[0] != 1.f) return false;
    const int M = x.i[0], F = y.i[1];
    const Bytes act = rows_of(p, y.t[1], M, F, 2);
    if (act.meets(operand_a(p, x)) || act.meets(operand_b(p, x)) || act.meets(result_c(p, x))) return false;
    return p.tensors[y.t[0]].offset == p.tensors[x.t[2]].offset && y.i[0] == M && 2 * F == x.i[1] && pitch(p, x.t[2]) == x.i[1] && pitch(p, y.t[1]) == F &&
           F % 128 != 0 && pair_swiglu_pays(M, F, x.i[2]);
}

// Whether two records next to each other are an attention backward and the inverse rotary embedding of its result. The table is read while other rows of
// the result are written, by pieces of 16 bytes (cai_rope_apply by 8).
inline bool backward_with_rotation(const Plan& p, const ExecOp& x, const ExecOp& y) {
    if (x.kernel != K_ATTN_BWD || y.kernel != K_ROPE || (x.flags && x.flags != 7) || !(y.flags & 1)) return false;
    if (!has_tensor(p, x.t[5]) || !has_tensor(p, y.t[0]) || !has_tensor(p, y.t[1])) return false;
    const Bytes table = tensor_bytes(p, y.t[1]), result = tensor_bytes(p, x.t[5]);
    if ((table.lo & 15) || table.meets(result)) return false;
    // B, S, heads of the one; rows, S, heads of the other, over rows of the same pitch
    return p.tensors[x.t[5]].offset == p.tensors[y.t[0]].offset && y.i[0] == x.i[0] * x.i[1] && y.i[1] == x.i[1] && y.i[2] == x.i[2] && y.i[3] == x.i[3] &&
           y.i[4] == x.i[4] && pitch(p, y.t[0]) == static_cast<long long>(x.i[2] + 2 * x.i[3]) * x.i[4];
}

// Products whose results no record of the plan reads: with activation recompute, the down projection of a layer that is run again for its
// backward. Nothing that any record names may lie in the bytes of a result for it to count as unread, outputs of plain bf16 products apart, and no
// tensor that the plan gives a name to. Only activations: other ranks read some of the rest, by records of their own.
inline void find_unread(const Plan& p, std::vector<uint8_t>* join) {
    auto product = [](const ExecOp& x) { return plain_product(x) && (epilogue(x) == CAI_EPI_BF16 || epilogue(x) == CAI_EPI_BF16_RESIDUAL); };
    std::vector<Bytes> used;
    for (const NamedTensor& n : p.named)
        for (const int t : {n.tensor, n.grad})
            if (has_tensor(p, t)) used.push_back(tensor_bytes(p, t));
    for (const ExecOp& x : p.exec)
        for (int k = 0; k < static_cast<int>(sizeof x.t / sizeof x.t[0]); ++k)
            if (has_tensor(p, x.t[k]) && !(k == 2 && product(x))) used.push_back(tensor_bytes(p, x.t[k]));
    std::sort(used.begin(), used.end(), [](const Bytes& a, const Bytes& b) { return a.lo < b.lo; });
    std::vector<uint64_t> reach(used.size());      // the furthest end of the ranges up to this one
    for (size_t i = 0; i < used.size(); ++i) reach[i] = i && reach[i - 1] > used[i].hi ? reach[i - 1] : used[i].hi;
    for (size_t i = 0; i < p.ops.size(); ++i) {
        if (!p.ops[i].exec || !product(p.exec[p.ops[i].exec - 1])) continue;
        const int result = p.exec[p.ops[i].exec - 1].t[2];
        if (!has_tensor(p, result) || p.tensors[result].tclass != TC_ACTIVATION) continue;
        const Bytes r = tensor_bytes(p, result);
        const size_t n = std::lower_bound(used.begin(), used.end(), r.hi, [](const Bytes& a, uint64_t hi) { return a.lo < hi; }) - used.begin();
        if (n == 0 || reach[n - 1] <= r.lo) (*join)[i] = kUnread;
    }
}

// Per record of the op table; a record that goes out with the one before it stays kAlone, and the walk does not come to it.
inline std::vector<uint8_t> find_joins(const Plan& p) {
    std::vector<uint8_t> join(p.ops.size() + 1, kAlone);
    find_unread(p, &join);
    for (size_t i = 0; i + 1 < p.ops.size(); ++i) {
        if (join[i] == kUnread || join[i + 1] == kUnread || !neighbours(p.ops[i], p.ops[i + 1])) continue;
        const ExecOp &x = p.exec[p.ops[i].exec - 1], &y = p.exec[p.ops[i + 1].exec - 1];
        join[i] = independent_products(p, x, y)     ? kPairOfProducts
                  : projection_with_swiglu(p, x, y) ? kWithSwiglu
                  : backward_with_rotation(p, x, y) ? kWithRotation
                                                    : kAlone;
        if (join[i] != kAlone) ++i;
    }
    return join;
}

// Sums of gain gradients that are still to go out (RMSNorm backward without its last step): they wait for each other in the rows of the plan's scratch
// that one norm leaves free, and go out before anything that could name what they read or write. A chain of short kernels is some 5 us shorter for each
// launch less: a step of 47 launches 298 -> 288 us, 8 layers of 896 tokens, three times over, 3632 -> 3519; 3840 tokens, where two norms fit, no change.
struct WaitingSums {
    struct Sum {
        uint64_t partial;      // offset in the arena of its partial rows
        int dg, parts, accumulate;
    };
    Sum sum[CAI_DG_SUMS];
    int n = 0, H = 0, stream = 0;
    Bytes scratch;             // the whole scratch
    uint64_t next = 0;         // its first free row

    // Must they go out before this operation? Those that only name tensors of their own record are looked at by range; others (whole
    // buffers, other ranks, other streams) and events count as naming everything.
    bool before(const Plan& p, const Op& op) const {
        if (!n) return false;
        if (op.kind == OP_EVENT_RECORD || op.kind == OP_EVENT_WAIT) return true;
        if (!op.exec) return false;
        if (op.stream_id != stream) return true;
        const ExecOp& x = p.exec[op.exec - 1];
        switch (x.kernel) {
            case K_GEMM: case K_GEMM_FP8: case K_QUANT_FP8: case K_SWIGLU_FWD: case K_SWIGLU_BWD: case K_ATTN_FWD: case K_ATTN_BWD: case K_ROPE:
            case K_RMSNORM_FWD: case K_RMSNORM_BWD: case K_EMBED_FWD: case K_EMBED_BWD: case K_CROSS_ENTROPY: case K_ADD: break;
            default: return true;
        }
        for (int k = 0; k < static_cast<int>(sizeof x.t / sizeof x.t[0]); ++k) {
            if (x.t[k] < 0 || (x.kernel == K_RMSNORM_BWD && k == 6)) continue;       // (the scratch itself: add() looks after its rows)
            const Bytes b = tensor_bytes(p, x.t[k]);
            if (b.meets(scratch)) return true;
            for (int i = 0; i < n; ++i) {
                const uint64_t dg = p.tensors[sum[i].dg].offset;
                if (b.meets({dg, dg + static_cast<uint64_t>(H) * sizeof(float)})) return true;
            }
        }
        return false;
    }
    // Room for the partial rows of a norm's sum beside those that wait: takes it, or says that they have to go out first.
    bool add(const Plan& p, const Op& op, const ExecOp& x, int parts) {
        const uint64_t need = static_cast<uint64_t>(parts) * x.i[1] * sizeof(float);
        const Bytes all = tensor_bytes(p, x.t[6]);
        if (!n) {
            H = x.i[1];
            stream = op.stream_id;
            scratch = all;
            next = all.lo;
        } else if (n == CAI_DG_SUMS || x.i[1] != H || op.stream_id != stream || all.lo != scratch.lo || next + need > scratch.hi) {
            return false;
        }
        sum[n++] = {next, x.t[5], parts, x.i[3]};
        next += need;
        return true;
    }
};

struct Launch {
    enum What : uint8_t { kEvent, kRecord, kTwoProducts, kSwiglu, kRotated, kNormSweep, kNormSums } what;
    uint32_t op;                    // the (first) operation; of kNormSums the one before which they go out
    const WaitingSums* sums;        // kNormSweep: its own is the last one; kNormSums: they go out
};

// The list, one at a time. join: what may be joined (false: every record by itself, as traced and checked replays launch it); products: also with products
// in other forms than those of single records (false under a limit on the SMs).
class LaunchWalk {
public:
    LaunchWalk(const Plan& plan, const std::vector<uint8_t>& joins, bool join, bool products, int sms)
        : p_(plan), joins_(joins), join_(join), products_(products), sms_(sms) {}
    bool next(Launch* l) {
        for (; at_ < p_.ops.size(); ++at_) {
            const Op& op = p_.ops[at_];
            const uint8_t how = joins_[at_];
            const bool two = how == kPairOfProducts || how == kWithSwiglu || how == kWithRotation;
            if (waiting_.before(p_, op) || (two && waiting_.before(p_, p_.ops[at_ + 1]))) return sums(l);
            if (op.kind == OP_EVENT_RECORD || op.kind == OP_EVENT_WAIT) return one(l, Launch::kEvent, 1);
            if (!op.exec) continue;
            const ExecOp& x = p_.exec[op.exec - 1];
            if (how == kUnread && join_ && !gather_) continue;
            // (a product that carries a gather writes more than its record names: behind a gather no sum waits)
            if (x.kernel == K_RMSNORM_BWD && join_ && !gather_) {
                const int parts = rmsnorm_partial_rows(x.i[0], x.i[1], sms_);
                const bool form = parts > 0 && has_tensor(p_, x.t[5]) && static_cast<uint64_t>(parts) * x.i[1] * sizeof(float) <= tensor_bytes(p_, x.t[6]).hi - tensor_bytes(p_, x.t[6]).lo;
                if (form && waiting_.add(p_, op, x, parts)) {
                    l->sums = &waiting_;
                    return one(l, Launch::kNormSweep, 1);
                }
                if (waiting_.n) return sums(l);      // no room left; or the whole form, which uses the scratch from its beginning
            }
            if (two && join_ && products_ && !gather_)
                return one(l, how == kPairOfProducts ? Launch::kTwoProducts : how == kWithSwiglu ? Launch::kSwiglu : Launch::kRotated, 2);
            // ZeRO-3: a gather rides in the next product
            if (x.kernel == K_FSDP_AG_GEMM && (x.flags & 1)) gather_ = true;
            if (x.kernel == K_GEMM) gather_ = false;
            return one(l, Launch::kRecord, 1);
        }
        return waiting_.n ? sums(l) : false;
    }

private:
    bool one(Launch* l, Launch::What what, uint32_t ops) {
        l->what = what;
        l->op = static_cast<uint32_t>(at_);
        at_ += ops;
        return true;
    }
    bool sums(Launch* l) {
        out_ = waiting_;
        waiting_.n = 0;
        l->sums = &out_;
        return one(l, Launch::kNormSums, 0);
    }
    const Plan& p_;
    const std::vector<uint8_t>& joins_;
    const bool join_, products_;
    const int sms_;
    size_t at_ = 0;
    bool gather_ = false;
    WaitingSums waiting_, out_;
};

}  // namespace cai
