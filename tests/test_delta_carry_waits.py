"""The chain of chunks of the delta rule (csrc/delta_chunk.cu): what its warps do when a bounded wait gives up, as an explicit search over every order in which
they can run.  No warp may be left at a barrier.  The order of the barriers and whose word is read where come from the kernel's source."""
import itertools
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "lit_gpt_b200", "csrc", "delta_chunk.cu")


def _link():
    """One chunk as its warps see it: "wait", "sync", "leave" (where the word is read); and whether every group has a word of its own."""
    text = open(SRC).read()
    body = text[text.index("for (int c = 0; c < chunks; ++c) {") : text.index("if (!ok) {")]
    ops = []
    for m in re.finditer(r"mbar_wait\(full.*?s_gave_up(\[group\])? = 1|group_sync\(\)|if \(\*\(volatile int\*\)&s_gave_up(\[group\])?\) \{ ok = false; break; \}", body):
        ops.append("wait" if m.group(0).startswith("mbar") else "sync" if m.group(0).startswith("group_sync") else "leave")
    assert ops == ["wait", "sync", "leave", "sync", "sync"] and len(re.findall("s_gave_up", body)) == 2
    return ops, len(re.findall(r"s_gave_up\[group\]", body)) == 2


def _stuck(groups, chunks, ops, own):
    """Whether some order leaves a warp at a barrier for good.  Two warps a group; any wait may give up, once in all (a copy that never comes)."""
    n = 2 * groups
    start = ((0,) * n, (0,) * groups, False)   # a warp's place (-1: it has left), the words, whether a wait gave up
    seen, todo = {start}, [start]
    end = chunks * len(ops)
    while todo:
        at, words, gave = todo.pop()
        nxt = []
        for w in range(n):
            p = at[w]
            if p < 0 or p == end:
                continue
            g = w // 2
            op = ops[p % len(ops)]
            move = lambda to, words=words, gave=gave: nxt.append((at[:w] + (to,) + at[w + 1 :], words, gave))   # noqa: E731,B023
            if op == "wait":
                move(p + 1)
                if not gave:
                    i = g if own else 0
                    move(p + 1, words[:i] + (1,) + words[i + 1 :], True)
            elif op == "leave":
                move(-1 if words[g if own else 0] else p + 1)
            else:   # both of the group's warps pass together
                mate = w ^ 1
                if at[mate] == p and mate > w:
                    a = list(at)
                    a[w] = a[mate] = p + 1
                    nxt.append((tuple(a), words, gave))
        if not nxt and any(0 <= p < end for p in at):
            return True
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return False


def test_search_finds_a_shared_word():
    ops = ["wait", "sync", "leave", "sync", "sync"]
    assert _stuck(2, 2, ops, False) and not _stuck(1, 3, ops, False)


@pytest.mark.parametrize("groups,chunks", list(itertools.product((1, 2), (1, 3))))
def test_no_warp_left_at_a_barrier(groups, chunks):
    ops, own = _link()
    assert not _stuck(groups, chunks, ops, own)
