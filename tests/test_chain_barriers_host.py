"""The barriers between the two warps of a SHA-256 chain pair (sha256.cuh: one warp runs
the rounds, the other the schedule), read from the source and run through every
interleaving: each use of a barrier brings together one arrival of each warp, of the
same place in the chain, no warp waits for ever, and the CTA's own barrier, which all
threads have to reach by the same instruction, stands in neither warp's code."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "truepix_b200", "csrc", "sha256.cuh")
OP = re.compile(r"\b(bar_arrive|bar_wait)\((\w+)\)")


def body(name):
    text = open(SRC).read()
    at = text.index(" %s(" % name, text.index("struct ChainMem"))
    return text[at:text.index("\n}", at)]


def operations(name, hashes):
    """(waits?, barrier) in the order in which the warp meets them"""
    head, loop = body(name).split("for (int n = 0; n < hashes; ++n) {")
    out = [(m[1] == "bar_wait", m[2]) for m in OP.finditer(head)]
    for n in range(hashes):
        inside = False                       # a block for all hashes but the last
        for line in loop.split("\n"):
            if "if (n + 1 < hashes) {" in line:
                inside = True
            elif line == "        }":
                inside = False
            for m in OP.finditer(line):
                if (inside and n + 1 == hashes) or ("if (n > 0)" in line and n == 0):
                    continue
                out.append((m[1] == "bar_wait", m[2]))
    return out


def test_no_barrier_of_the_whole_cta():
    for name in ("chain_rounds", "chain_schedule", "chain_pair"):
        assert "__syncthreads" not in body(name), name


@pytest.mark.parametrize("hashes", [1, 2, 3, 64])
def test_every_interleaving(hashes):
    progs = [operations(n, hashes) for n in ("chain_rounds", "chain_schedule")]
    uses = [{}, {}]
    for w in (0, 1):                         # the ordinal of each use of a barrier by its warp
        for i, (_, b) in enumerate(progs[w]):
            uses[w][i] = (b, sum(1 for _, q in progs[w][:i] if q == b))
    assert {b for _, b in progs[0]} == {b for _, b in progs[1]} == {"kBarH", "kBarA", "kBarB", "kBarC", "kBarPair"}
    # a state: next operation of each warp, the barriers with one arrival (its warp and
    # operation), and the barrier each warp is held at
    start = (0, 0, frozenset(), None, None)
    seen, todo = {start}, [start]
    while todo:
        pc0, pc1, pending, held0, held1 = todo.pop()
        pc, held = [pc0, pc1], [held0, held1]
        able = [w for w in (0, 1) if held[w] is None and pc[w] < len(progs[w])]
        if not able:
            assert pc == [len(p) for p in progs] and held == [None, None] and not pending, "held for ever"
        for w in able:
            waits, b = progs[w][pc[w]]
            there = {q: (v, i) for q, v, i in pending}
            n_pc, n_held = list(pc), list(held)
            n_pc[w] += 1
            if b in there:
                v, i = there.pop(b)
                assert v != w and uses[v][i] == uses[w][pc[w]], "two uses of %s meet" % b
                if n_held[v] == b:
                    n_held[v] = None
            else:
                there[b] = (w, pc[w])
                if waits:
                    n_held[w] = b
            state = (n_pc[0], n_pc[1], frozenset((q, v, i) for q, (v, i) in there.items()), n_held[0], n_held[1])
            if state not in seen:
                seen.add(state)
                todo.append(state)
