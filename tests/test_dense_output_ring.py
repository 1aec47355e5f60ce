"""The hand-over of the row tiles' outputs in the dense forward, followed through every interleaving of its warps.

A model of csrc/dense_fwd_tc.cu: the loads, the warp that issues the products, the two softmax groups and the warp that stores the
outputs, over items of one key tile each, with the barriers that stand between them.  Which o_full barrier a tile uses, and the parity
that is waited for, are taken from the source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "native_sparse_attention_triton_b200", "csrc", "dense_fwd_tc.cu")
BUFS = 3


def _expressions():
    text = open(SOURCE).read()
    assert re.search(r"kTcQBufs = %d;" % BUFS, text)
    waits = re.findall(r"mbar_wait\(o_full \+ (.+?), (.+?), p\.st\);", text)
    arrivals = re.findall(r"mbar_arrive\(o_full \+ (.+?)\);", text)
    assert len(waits) == 1 and len(arrivals) == 1
    return waits[0] + (arrivals[0],)


def _value(expr, tile):
    return int(eval(expr.replace("/", "//"), {"rt": tile, "g": tile & 1, "qb": tile % BUFS, "kTcQBufs": BUFS}))


def _programs(items, seen_early):
    """Steps of each warp.  ("wait", barrier, parity) or ("arrive", barrier); a barrier completes one phase per arrival here.
    seen_early[i]: the issuing warp learns of item i + 1 before it issues the last product of item i."""
    wait_slot, wait_parity, arrive_slot = _expressions()
    tiles = 2 * items
    load = []
    for t in range(tiles):
        if t >= BUFS:
            load.append(("wait", f"q_empty{t % BUFS}", (t // BUFS - 1) & 1))
        load.append(("arrive", f"q_full{t % BUFS}"))
    issue = []

    def start(t):
        issue.extend([("wait", f"q_full{t % BUFS}", (t // BUFS) & 1), ("arrive", f"s_full{t & 1}")])

    def product(t):
        issue.extend([("wait", f"p_full{t & 1}", (t >> 1) & 1), ("arrive", f"pv_done{t & 1}")])

    start(0)
    start(1)
    for i in range(items):
        last = i + 1 == items
        product(2 * i)
        if not last and seen_early[i]:
            start(2 * i + 2)
        product(2 * i + 1)
        if not last:
            if not seen_early[i]:
                start(2 * i + 2)
            start(2 * i + 3)
    softmax = [[], []]
    for t in range(tiles):
        softmax[t & 1] += [("wait", f"s_full{t & 1}", (t >> 1) & 1), ("arrive", f"p_full{t & 1}"), ("wait", f"pv_done{t & 1}", (t >> 1) & 1),
                           ("arrive", f"o_full{_value(arrive_slot, t)}")]
    store = []
    for t in range(tiles):
        store += [("wait", f"o_full{_value(wait_slot, t)}", _value(wait_parity, t)), ("arrive", f"q_empty{t % BUFS}")]
    return [load, issue, *softmax, store]


@pytest.mark.parametrize("seen_early", [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)])
def test_every_interleaving_ends(seen_early):
    programs = _programs(len(seen_early) + 1, seen_early)
    names = sorted({step[1] for prog in programs for step in prog})
    at = {n: i for i, n in enumerate(names)}
    begin = ((0,) * len(programs), (0,) * len(names))
    todo, known = [begin], {begin}
    while todo:
        pcs, phases = todo.pop()
        moved = False
        for w, prog in enumerate(programs):
            if pcs[w] == len(prog):
                continue
            step = prog[pcs[w]]
            now = phases
            if step[0] == "wait":
                if phases[at[step[1]]] & 1 == step[2]:   # the phase of that parity has not completed, or the one after it has too
                    continue
            else:
                b = at[step[1]]
                now = phases[:b] + ((phases[b] + 1) % 4,) + phases[b + 1:]
            moved = True
            state = (pcs[:w] + (pcs[w] + 1,) + pcs[w + 1:], now)
            if state not in known:
                known.add(state)
                todo.append(state)
        stuck = [prog[pc] for pc, prog in zip(pcs, programs) if pc < len(prog)]
        assert moved or not stuck, f"no warp can go on: {stuck}"
