"""The barrier protocol of the FP8 attention kernel, walked through in every order of events (CPU).

One TMA producer, two MMA issuers and the softmax warps meet on mbarriers whose waits look at the parity of a phase
only.  Such a wait is sound as long as the barrier can be at most one completed phase ahead of the waiter: two ahead
reads as "not yet" and the wait never ends.  The model below has the threads' waits, arrivals, loads and commits in the
order in which csrc/attention.cu issues them; loads land and commits arrive at any later time (each issuer's commits in
their order).  The search visits every reachable state.
"""
import collections

import pytest

SLOTS = 3          # kAttnKS


def _programs(nblk, multi, tiles, shared_slot_barrier, warps=2):
    slot_free = (lambda i: (("slot_free", 0), i)) if shared_slot_barrier else (lambda i: (("slot_free", i % SLOTS), i // SLOTS))
    load = lambda *b: ("load", b)
    wait = lambda b, k: ("wait", b, k)
    commit = lambda b: ("commit", b)
    s_full, step_end = ("s_full",), ("step_end",)
    producer = [load("q", 0)]
    for j in range(min(nblk, SLOTS)):
        producer += [load("k", j), load("v", j)]
    if multi:
        producer += [load("q", 1)] if tiles > 1 else []
        for t in range(tiles - 2):
            producer += [wait(("q_free", t & 1), t >> 1), load("q", t & 1)]
    else:
        for i in range(nblk - SLOTS):
            producer += [wait(*slot_free(i)), load("k", i % SLOTS), load("v", i % SLOTS)]
    pv, qk, softmax = [], [], []
    for t in range(tiles):
        e = t * (nblk + 2) if multi else 0
        if t > 0:
            pv.append(wait(step_end, e - 1))
            qk.append(wait(step_end, e - 1))
        pv += [commit(s_full), wait(step_end, e), commit(s_full)]
        for i in range(nblk):
            pv += [wait(step_end, e + i + 1), wait(("v", i % SLOTS), i // SLOTS), commit(s_full)]
            if not multi and i + SLOTS < nblk:
                pv.append(commit(slot_free(i)[0]))
        if multi and t + 2 < tiles:
            pv.append(commit(("q_free", t & 1)))
        qk += [wait(("q", t & 1), t >> 1), wait(("k", 0), 0), commit(s_full), wait(step_end, e)]
        qk += [wait(("k", 1), 0)] if nblk > 1 else []
        qk.append(commit(s_full))
        for i in range(nblk):
            qk.append(wait(step_end, e + i + 1))
            if i + 2 < nblk:
                qk.append(wait(("k", (i + 2) % SLOTS), (i + 2) // SLOTS))
            qk.append(commit(s_full))
        softmax += [wait(s_full, e), ("arrive", step_end)]
        for i in range(nblk):
            softmax += [wait(s_full, e + i + 1), ("arrive", step_end)]
        softmax.append(wait(s_full, e + nblk + 1))
        if multi:
            softmax.append(("arrive", step_end))
    return [producer, pv, qk] + [softmax] * warps, {s_full: 2, step_end: warps}


def _search(programs, arrivals_per_phase):
    """Faults found: waits that a barrier has left two phases behind or lets through a phase early, and dead ends."""
    start = (tuple(0 for _ in programs), (), (), (), ())
    seen, todo, faults = {start}, collections.deque([start]), set()
    while todo:
        pcs, arrived, pv_fifo, qk_fifo, loads = todo.popleft()
        count = dict(arrived)

        def plus(bar):
            return tuple(sorted({**count, bar: count.get(bar, 0) + 1}.items()))

        succ = []
        for t, prog in enumerate(programs):
            if pcs[t] == len(prog):
                continue
            op = prog[pcs[t]]
            after = pcs[:t] + (pcs[t] + 1,) + pcs[t + 1:]
            if op[0] == "wait":
                done = count.get(op[1], 0) // arrivals_per_phase.get(op[1], 1)
                passes = done % 2 != op[2] % 2
                if done > op[2] + 1 or (passes and done <= op[2]):
                    faults.add((t, op[1]))
                if passes:
                    succ.append((after, arrived, pv_fifo, qk_fifo, loads))
            elif op[0] == "arrive":
                succ.append((after, plus(op[1]), pv_fifo, qk_fifo, loads))
            elif op[0] == "load":
                succ.append((after, arrived, pv_fifo, qk_fifo, tuple(sorted(loads + (op[1],)))))
            elif t == 1:
                succ.append((after, arrived, pv_fifo + (op[1],), qk_fifo, loads))
            else:
                succ.append((after, arrived, pv_fifo, qk_fifo + (op[1],), loads))
        if pv_fifo:
            succ.append((pcs, plus(pv_fifo[0]), pv_fifo[1:], qk_fifo, loads))
        if qk_fifo:
            succ.append((pcs, plus(qk_fifo[0]), pv_fifo, qk_fifo[1:], loads))
        for i, bar in enumerate(loads):
            succ.append((pcs, plus(bar), pv_fifo, qk_fifo, loads[:i] + loads[i + 1:]))
        if not succ and any(pc < len(prog) for pc, prog in zip(pcs, programs)):
            faults.add("dead end")
        for s in succ:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return faults


@pytest.mark.parametrize("nblk,multi,tiles", [(n, False, 1) for n in (1, 2, 3, 4, 5, 7, 8)] + [(n, True, 4) for n in (1, 2, 3)])
def test_every_order_of_events_ends(nblk, multi, tiles):
    assert _search(*_programs(nblk, multi, tiles, shared_slot_barrier=False)) == set()


def test_one_barrier_for_all_slots_would_not():
    """The model sees the fault that separate slot barriers rule out: a producer held up for one step."""
    faults = _search(*_programs(6, False, 1, shared_slot_barrier=True))
    assert "dead end" in faults and (0, ("slot_free", 0)) in faults
