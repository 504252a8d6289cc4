"""Hand-over of the reference maximum between the two softmax teams of the prefill attention, on the CPU.

Four warps share a quarter of the query rows: two teams (alternate key blocks) of two column halves.  Every order in which
they can run is tried on a model of the mbarrier that publishes a block's reference (two arrivals a phase; a wait for a
parity passes unless the current phase has it) and of the named barriers.  What the warps do after their last block is
read from the kernel's source, in its order."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tokenselect_b200", "csrc", "extend.cu")


def _tail_ops():
    text = open(SOURCE).read()
    body = text[text.index("extend_attend_tc5_wide_kernel(const ExtendParams e)"):]
    tail = re.sub(r"//[^\n]*", "", body[body.index("// row sums:"):body.index("const float l_tot")])
    kinds = {"mbar_wait(smem_u32(&sm.ref_ready": "wait", "named_bar_sync(9": "quarter", "sm.ref[(nblk - 1)": "read"}
    found = sorted((m.start(), kind) for pat, kind in kinds.items() for m in re.finditer(re.escape(pat), tail))
    assert "read" in [kind for _, kind in found]
    return [kind for _, kind in found]


def _program(team, half, nblk, tail):
    ops = []
    for blk in range(team, nblk, 2):
        ops.append(("team", blk))                               # the named barrier of the row maxima
        if blk > 0:
            ops += [("wait", (blk - 1) & 1), ("read", blk - 1)]
        if half == 0:
            ops.append(("write", blk))
        ops.append(("arrive", blk))
    for i, kind in enumerate(tail):
        ops.append({"wait": ("wait", (nblk - 1) & 1), "read": ("read", nblk - 1), "quarter": ("quarter", i)}[kind])
    return ops


def _faults(nblk, tail):
    progs = [_program(team, half, nblk, tail) for team in (0, 1) for half in (0, 1)]
    faults, seen = set(), set()
    todo = [((0, 0, 0, 0), 0, 0, (None, None))]                 # program counters, arrivals, phase, the two references
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        pc, arrived, phase, ref = state
        moved = False
        for w in range(4):
            if pc[w] == len(progs[w]):
                continue
            kind, arg = progs[w][pc[w]]
            go, a, ph, r = [w], arrived, phase, ref
            if kind == "wait" and (phase & 1) == arg:
                continue
            if kind == "read" and ref[arg & 1] != arg:
                faults.add(("stale reference", w, arg, ref[arg & 1]))
            if kind == "write":
                r = tuple(arg if i == (arg & 1) else ref[i] for i in (0, 1))
            if kind == "arrive":
                a, ph = (0, phase + 1) if arrived == 1 else (arrived + 1, phase)
            if kind in ("team", "quarter"):
                go = [x for x in range(4) if kind == "quarter" or x // 2 == w // 2]
                if any(pc[x] == len(progs[x]) or progs[x][pc[x]] != (kind, arg) for x in go):
                    continue
            moved = True
            todo.append((tuple(pc[x] + (x in go) for x in range(4)), a, ph, r))
        if not moved and any(pc[w] < len(progs[w]) for w in range(4)):
            faults.add(("stuck", pc))
    return faults


@pytest.mark.parametrize("nblk", [1, 2, 3, 4, 5, 6])
def test_every_order_reads_the_published_reference(nblk):
    assert not _faults(nblk, _tail_ops())


def test_the_model_sees_a_wait_without_the_barrier():
    assert _faults(2, ["wait", "read", "quarter"])
