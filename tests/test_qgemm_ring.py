"""Prompt GEMM (csrc/qgemm.cu): the ring of packed weights between the warp that fetches them and the two groups of dequantising warps, as an explicit search
over every order in which the barriers let warps run.  No buffer may be written before all of its readers are done.  The ring's sizes and what a group does
about a last pair of k-blocks whose second half does not exist are read from the kernel's source."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "lit_gpt_b200", "csrc", "qgemm.cu")


def _ring():
    text = open(SRC).read()
    mt2, mt1 = map(int, re.search(r"kStages = MT == 2 \? (\d+) : (\d+);", text).groups())
    buffers = int(re.search(r"kPairs = (\d+)", text).group(1))
    # the statement that stands in for the missing block: from its condition to the next line of the common path
    last = re.search(r"if \(\(t\.nkb & 1\) && l0 == 1.*?pairs \+= \(t\.nkb \+ 1\) >> 1;", text, re.S).group(0)
    assert last.count("mbar_arrive(w_empty") == 1
    waits = re.search(r"mbar_wait\(w_full.*mbar_arrive\(w_empty", last, re.S) is not None
    return {1: mt1, 2: mt2}, buffers, waits


def _programs(items, stages, waits):
    """What a warp of either group does, in order: ("full", pair), ("read", pair), ("room", block), ("empty", pair), ("block", block), ("done", blocks)."""
    out = ([], [])
    q = pairs = 0
    for nkb in items:
        for g in (0, 1):
            l0 = (g + q) % 2
            for l in range(l0, nkb, 2):
                p = pairs + l // 2
                out[g].extend([("full", p), ("read", p), ("room", q + l), ("empty", p), ("block", q + l)])
            if nkb % 2 and l0 == 1:
                p = pairs + nkb // 2
                out[g].extend(([("full", p)] if waits else []) + [("empty", p)])
        pairs += (nkb + 1) // 2
        q += nkb
        for g in (0, 1):
            out[g].append(("done", q))
    return out, pairs, q


def _overwritten(items, stages, buffers, waits):
    """A pair whose buffer can be written over before a warp has read it, or None.  Two warps a group: one that runs on and one that is held up anywhere."""
    programs, pairs, blocks = _programs(items, stages, waits)
    prog = (programs[0], programs[0], programs[1], programs[1])
    ops = [[sum(1 for op in w[:i] if op[0] == "empty" and op[1] % buffers == b) for i in range(len(w) + 1)] for w in prog for b in range(buffers)]
    wrote = [{op[1]: i + 1 for i, op in enumerate(w) if op[0] == "block"} for w in prog]
    reads = [{} for _ in prog]
    for w, r in zip(prog, reads):
        for i, op in enumerate(w):
            if op[0] == "read":
                r[op[1]] = i + 1   # (the last of a pair's reads by this warp)
    start = ((0, 0, 0, 0), 0, 0)   # warps, pairs fetched, blocks multiplied
    seen, todo = {start}, [start]
    while todo:
        at, fetched, used = todo.pop()
        nxt = []
        if fetched < pairs:
            b = fetched % buffers
            if sum(ops[w * buffers + b][at[w]] for w in range(4)) >= 4 * (fetched // buffers):   # the phase before this one is complete
                if fetched >= buffers and any(at[w] < reads[w].get(fetched - buffers, 0) for w in range(4)):
                    return fetched - buffers
                nxt.append((at, fetched + 1, used))
        if used < blocks and all(at[w] >= wrote[w][used] for w in range(4) if used in wrote[w]):
            nxt.append((at, fetched, used + 1))
        for w in range(4):
            if at[w] < len(prog[w]):
                what, n = prog[w][at[w]]
                if what == "full" and n >= fetched or what == "room" and used < n - stages + 1 or what == "done" and used < n:
                    continue
                nxt.append((at[:w] + (at[w] + 1,) + at[w + 1 :], fetched, used))
        if not nxt:
            assert fetched == pairs and used == blocks and all(at[w] == len(prog[w]) for w in range(4)), "the barriers wait for one another"
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def test_ring_search_finds_an_early_release():
    assert _overwritten((9,), 6, 3, False) is not None and _overwritten((8,), 6, 3, False) is None and _overwritten((9,), 4, 3, False) is None


@pytest.mark.parametrize("items", [(1, 1, 3), (7,), (8,), (9,), (11,), (5, 7), (7, 4)])
@pytest.mark.parametrize("mt", [1, 2])
def test_ring_never_written_early(items, mt):
    stages, buffers, waits = _ring()
    assert _overwritten(items, stages[mt], buffers, waits) is None
