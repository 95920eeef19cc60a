"""What a replay of a plan launches: records that go out together, results left out, sums that wait. Which ones follows from the plan alone, so it is asked
here, where there is no GPU, for the layouts that several GPUs run as well."""
import ctypes
from pathlib import Path

import pytest
import torch

from cai_b200 import plan as planlib
from cai_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib._LIB_PATH.exists(), reason="kernel library not built")

ROOT = Path(__file__).resolve().parent.parent
EVENT, RECORD, TWO_PRODUCTS, SWIGLU, ROTATED, NORM_SWEEP, NORM_SUMS = range(7)
K = {n: i for i, n in enumerate(planlib.KERNEL_NAMES)}
EVENTS = (planlib.OP_EVENT_RECORD, planlib.OP_EVENT_WAIT)


def launches(raw, join=1):
    """(what, first operation, sums that go out, kernels) of every launch."""
    ask = lambda buf, n: _lib.lib().cai_plan_launches(ctypes.c_char_p(raw), ctypes.c_size_t(len(raw)), join, buf, n)
    n = ask(None, 0)
    assert n >= 0, _lib.lib().cai_last_error()
    buf = (ctypes.c_int * (4 * max(n, 1)))()
    assert ask(buf, n) == n
    return [tuple(buf[4 * i:4 * i + 4]) for i in range(n)]


def config(base, world, keys=""):
    return ((ROOT / "configs" / base).read_text() +
            f"\ngpus_per_rack = {world}\ngpus_per_tray = {world}\ntrays_per_rack = 1\nnum_racks = 1\n{keys}\n")


def plans(tmp_path, base, world, keys=""):
    planlib.compile_plans(config(base, world, keys), tmp_path, ranks=(0, world), version=2, text=True)
    return [planlib.PlanFile(tmp_path / f"plan.rank{r:06d}.bin") for r in range(world)]


ODD = "hidden_size = 1000\nffn_hidden = 2728\nvocab_size = 5000\nseq_len = 640\nmicrobatch = 3\n"
LAYOUTS = {      # base, ranks, keys, what has to be among the launches of some rank
    "one rank": ("tiny.cfg", 1, "", {TWO_PRODUCTS, ROTATED, NORM_SWEEP}),
    "one rank, odd widths": ("tiny.cfg", 1, ODD, {TWO_PRODUCTS, SWIGLU, ROTATED}),
    "one rank, odd widths, recompute": ("tiny.cfg", 1, ODD + "recompute = 1", {TWO_PRODUCTS, SWIGLU, ROTATED, "unread"}),
    "one rank, e4m3, recompute": ("tiny.cfg", 1, "param_dtype = fp8e4m3\nrecompute = 1", {ROTATED, NORM_SWEEP}),
    "one rank, experts": ("tiny_moe.cfg", 1, "", {ROTATED, NORM_SWEEP}),
    "tp2": ("tiny_mp.cfg", 2, "tp = 2\ncomm = fused", set()),
    "tp2, recompute": ("tiny_mp.cfg", 2, "tp = 2\ncomm = fused\nrecompute = 1", set()),
    "tp2, serial weight gradients": ("tiny_mp.cfg", 2, "tp = 2\ncomm = fused\nwgrad_overlap = 0", {ROTATED}),
    "tp2, NCCL": ("tiny_mp.cfg", 2, "tp = 2\ncomm = baseline", set()),
    "pp2": ("tiny_mp.cfg", 2, "pp = 2\nrecompute = 1", {TWO_PRODUCTS, ROTATED, NORM_SWEEP, "unread"}),
    "dp2": ("tiny_mp.cfg", 2, "comm = fused", {TWO_PRODUCTS, ROTATED, NORM_SWEEP}),
    "dp2, NCCL": ("tiny_mp.cfg", 2, "comm = baseline", {TWO_PRODUCTS, ROTATED, NORM_SWEEP}),
    "dp2, ZeRO-2": ("tiny_mp.cfg", 2, "comm = fused\nzero_stage = 2\nmb_group = 1", {TWO_PRODUCTS, ROTATED, NORM_SWEEP}),
    "dp2, ZeRO-3": ("tiny_mp.cfg", 2, "comm = fused\nzero_stage = 3", {ROTATED, NORM_SWEEP}),
    "dp2, ZeRO-3, recompute": ("tiny_mp.cfg", 2, "comm = fused\nzero_stage = 3\nrecompute = 1", {ROTATED, NORM_SWEEP}),
    "tp2 x pp2 x dp2": ("tiny_mp.cfg", 8, "tp = 2\npp = 2\ncomm = fused", set()),
    "pp2 x dp2, ZeRO-3": ("tiny_mp.cfg", 4, "pp = 2\ncomm = fused\nzero_stage = 3", {ROTATED, NORM_SWEEP}),
    "experts over pp2 x ep2": ("tiny_moe.cfg", 4, "pp = 2\nep = 2\ncomm = fused", {ROTATED, NORM_SWEEP}),
}


def tensor_bytes(pf, t):
    return (pf.tensors[t].offset, pf.tensors[t].offset + pf.tensors[t].nbytes)


def meet(a, b):
    return a[0] < b[1] and b[0] < a[1]


@pytest.mark.parametrize("name", sorted(LAYOUTS))
def test_launches_cover_the_plan_and_keep_its_order(tmp_path, name):
    base, world, keys, expected = LAYOUTS[name]
    found = set()
    for pf in plans(tmp_path, base, world, keys):
        ops, steps = pf.ops, launches(pf.raw)
        record = lambda i: pf.exec[ops[i].exec - 1]
        # traced, every operation goes out by itself
        assert [(w, i) for w, i, _, _ in launches(pf.raw, 0)] == [(EVENT if op.kind in EVENTS else RECORD, i) for i, op in enumerate(ops)
                                                                 if op.exec or op.kind in EVENTS]
        covered, waiting, gather = [], [], False
        for what, i, sums, kernels in steps:
            found.add(what)
            if what == NORM_SUMS:
                assert 0 < sums == len(waiting) <= 8 and kernels == 1
                waiting = []
                continue
            mine = [i, i + 1] if what in (TWO_PRODUCTS, SWIGLU, ROTATED) else [i]
            covered += mine
            assert (what == EVENT) == (ops[i].kind in EVENTS)
            for j in mine:      # sums that wait, and what they read and write, are named by nothing until they have gone out
                for stream, scratch, dg in waiting:
                    assert ops[j].kind not in EVENTS and ops[j].stream_id == stream, (name, i)
                    norm = record(j).kernel == K["rmsnorm_bwd"]
                    for slot, t in enumerate(record(j).t):
                        if t >= 0:
                            assert not meet(tensor_bytes(pf, t), dg) and (norm and slot == 6 or not meet(tensor_bytes(pf, t), scratch)), (name, i, slot)
            if what == NORM_SWEEP:
                x = record(i)
                waiting.append((ops[i].stream_id, tensor_bytes(pf, x.t[6]), tensor_bytes(pf, x.t[5])))
            if len(mine) == 2:
                a, b = record(i), record(i + 1)
                assert not gather and ops[i].stream_id == ops[i + 1].stream_id and ops[i + 1].kind not in EVENTS
                if what == TWO_PRODUCTS:
                    assert a.kernel == b.kernel == K["gemm"] and kernels in (1, 2)
                    for x, y in ((a, b), (b, a)):      # neither touches what the other writes
                        assert not any(t >= 0 and meet(tensor_bytes(pf, t), tensor_bytes(pf, y.t[2])) for t in x.t[:4])
                elif what == SWIGLU:
                    assert a.kernel == K["gemm"] and b.kernel == K["swiglu_fwd"] and a.t[2] == b.t[0]
                else:
                    assert a.kernel == K["attn_bwd"] and b.kernel == K["rope"] and b.flags & 1 and a.t[5] == b.t[0]
            elif what == RECORD:      # a gather that waits rides in the next product
                gather = (gather or record(i).kernel == K["fsdp_ag_gemm"] and bool(record(i).flags & 1)) and record(i).kernel != K["gemm"]
        assert not waiting and not gather
        unread = [i for i, op in enumerate(ops) if (op.exec or op.kind in EVENTS) and i not in set(covered)]
        assert sorted(covered + unread) == [i for i, op in enumerate(ops) if op.exec or op.kind in EVENTS] and covered == sorted(covered)
        if unread:
            found.add("unread")
        others = [tensor_bytes(pf, t) for i, op in enumerate(ops) if op.exec for slot, t in enumerate(record(i).t) if t >= 0 and not (i in unread and slot == 2)]
        others += [tensor_bytes(pf, t) for n in pf.named for t in (n.tensor, n.grad) if t >= 0]
        for i in unread:
            assert record(i).kernel == K["gemm"] and not any(meet(tensor_bytes(pf, record(i).t[2]), o) for o in others)
    assert expected <= found, (name, found)


def _replayed(interp):
    """The interpreter's ranks issue what a replay launches: results that nothing reads left out, the second of two joined products first (neither may
    notice), gain gradients added up when their sums go out."""
    for r in interp.ranks:
        pf, r.sums_before, r.waiting, r.at = r.pf, set(), [], 0
        steps = launches(pf.raw)
        keep = set()
        for what, i, _, _ in steps:
            if what == NORM_SUMS:
                r.sums_before.add(i)
                continue
            keep |= {i, i + 1} if what in (TWO_PRODUCTS, SWIGLU, ROTATED) else {i}
            if what == TWO_PRODUCTS:
                a, b = pf.ops[i].exec, pf.ops[i + 1].exec
                pf.ops[i].exec, pf.ops[i + 1].exec = b, a
        for i, op in enumerate(pf.ops):
            op.flops = i                         # its place, for issue()
            if i not in keep:
                op.exec = 0
    issue, norm = interp._issue, interp._local[K["rmsnorm_bwd"]]

    def out(r):
        for dg, part in r.waiting:
            dg.copy_(part)
        r.waiting = []

    def delayed_norm(self, r, x):
        dg = r.flat(x.t[5], x.i[1])
        old = dg.clone()
        norm(self, r, x)
        r.waiting.append((dg, dg.clone()))
        dg.copy_(old)

    def replayed_issue(r, op, resumed=None):
        if resumed is None:
            while r.at <= op.flops:
                if r.at in r.sums_before:
                    out(r)
                r.at += 1
        return issue(r, op, resumed)

    step = interp.step

    def replayed_step(*args):
        for r in interp.ranks:
            r.at = 0
        loss = step(*args)
        for r in interp.ranks:
            out(r)
        return loss

    interp._local = {**interp._local, K["rmsnorm_bwd"]: delayed_norm}
    interp._issue, interp.step = replayed_issue, replayed_step
    return interp


@pytest.mark.parametrize("name", ["one rank", "one rank, e4m3, recompute", "tp2, recompute", "tp2, serial weight gradients", "pp2", "dp2", "dp2, ZeRO-2",
                                  "dp2, ZeRO-3, recompute", "pp2 x dp2, ZeRO-3", "experts over pp2 x ep2"])
def test_what_is_launched_trains_to_the_bits_of_the_plan(name):
    from cai_b200.models.plan_interpreter import PlanInterpreter, random_state
    base, world, keys, _ = LAYOUTS[name]
    text = config(base, world, keys)
    jobs = [PlanInterpreter(text), _replayed(PlanInterpreter(text))]
    st = random_state(jobs[0], seed=3)
    m, g = jobs[0].model, torch.Generator().manual_seed(5)
    rows = jobs[0].rows_per_replica * int(jobs[0].hdr.dp)
    batches = [torch.randint(0, m.vocab_size, (rows, int(m.seq_len)), generator=g) for _ in range(3)]
    losses = []
    for job in jobs:
        job.load_state(st)
        losses.append([job.step(batches[i], batches[i + 1]) for i in range(2)])
    assert losses[0] == losses[1]
    a, b = jobs[0].state(), jobs[1].state()
    for k in a:
        for key in ("master", "m", "v"):
            assert (a[k][key] == b[k][key]).all(), (name, k, key)


def moved(pf, t, **fields):
    """The plan's bytes with fields of tensor t's entry replaced."""
    raw = bytearray(pf.raw)
    at = ctypes.sizeof(planlib.PlanHeader) + t * ctypes.sizeof(planlib.TensorDesc)
    entry = planlib.TensorDesc.from_buffer_copy(raw, at)
    for k, v in fields.items():
        setattr(entry, k, v)
    raw[at:at + ctypes.sizeof(entry)] = bytes(entry)
    return bytes(raw)


def first(raw, what):
    return next((i for w, i, _, _ in launches(raw) if w == what), None)


# An activation that lies over what the product reads or writes is right where the records go out one behind the other.
@pytest.mark.parametrize("over", [0, 1, 2])
def test_swiglu_over_its_products_operands_goes_out_by_itself(tmp_path, over):
    pf, = plans(tmp_path, "tiny.cfg", 1, ODD)
    i = first(pf.raw, SWIGLU)
    x, y = (pf.exec[pf.ops[j].exec - 1] for j in (i, i + 1))
    lo, hi = tensor_bytes(pf, x.t[over])
    act = pf.tensors[y.t[1]].nbytes
    for at in (lo, hi - 512, max(lo - act + 512, 0)):      # over its beginning, its end, and with its own end
        if at + act <= pf.hdr.arena_bytes:
            assert (RECORD, i) in [(w, j) for w, j, _, _ in launches(moved(pf, y.t[1], offset=at))]


def test_rotation_whose_table_the_backward_cannot_take_goes_out_by_itself(tmp_path):
    pf, = plans(tmp_path, "tiny.cfg", 1)
    i = first(pf.raw, ROTATED)
    x, y = (pf.exec[pf.ops[j].exec - 1] for j in (i, i + 1))
    alone = lambda raw: {(RECORD, i), (RECORD, i + 1)} <= {(w, j) for w, j, _, _ in launches(raw)}
    table, (lo, hi) = pf.tensors[y.t[1]], tensor_bytes(pf, x.t[5])
    assert table.offset % 16 == 0 and not alone(pf.raw) and not alone(moved(pf, y.t[1], offset=table.offset + 16, nbytes=table.nbytes - 16))
    assert alone(moved(pf, y.t[1], offset=table.offset + 8, nbytes=table.nbytes - 8))      # 8 bytes are enough for the rotation by itself
    assert alone(moved(pf, y.t[1], offset=lo)) and alone(moved(pf, y.t[1], offset=hi - 512))


def test_only_activations_are_left_out(tmp_path):
    pf, = plans(tmp_path, "tiny.cfg", 1, ODD + "recompute = 1")

    def left_out(raw):
        covered = set()
        for what, i, _, _ in launches(raw):
            if what != NORM_SUMS:
                covered |= {i, i + 1} if what in (TWO_PRODUCTS, SWIGLU, ROTATED) else {i}
        return [i for i, op in enumerate(pf.ops) if op.exec and i not in covered]

    result = {pf.exec[pf.ops[i].exec - 1].t[2] for i in left_out(pf.raw)}
    assert len(result) == 1
    t, = result
    for tclass, name in enumerate(planlib.TCLASSES):
        assert bool(left_out(moved(pf, t, tclass=tclass))) == (name == "activation"), name


def test_no_sum_waits_behind_a_gather(tmp_path):
    """The product a gather rides in writes the gathered parameters, which its record does not name. The compiler puts it right behind the gather's record; here
    a norm comes in between."""
    pf = plans(tmp_path, "tiny_mp.cfg", 2, "comm = fused\nzero_stage = 3")[0]
    record = lambda i: pf.exec[pf.ops[i].exec - 1]
    gather = next(i for i, op in enumerate(pf.ops) if op.exec and record(i).kernel == K["fsdp_ag_gemm"] and record(i).flags & 1)
    assert record(gather + 1).kernel == K["gemm"]
    norm = next(i for i in range(gather, len(pf.ops)) if pf.ops[i].exec and record(i).kernel == K["rmsnorm_bwd"])
    assert (NORM_SWEEP, norm) in [(w, i) for w, i, _, _ in launches(pf.raw)] and pf.ops[norm].stream_id == pf.ops[gather].stream_id
    pf.ops[gather + 1].exec, pf.ops[norm].exec = pf.ops[norm].exec, pf.ops[gather + 1].exec
    at = ctypes.sizeof(planlib.PlanHeader) + ctypes.sizeof(pf.tensors) + ctypes.sizeof(pf.groups)
    steps = [(w, i) for w, i, _, _ in launches(pf.raw[:at] + bytes(pf.ops) + pf.raw[at + ctypes.sizeof(pf.ops):])]
    assert (RECORD, gather + 1) in steps
