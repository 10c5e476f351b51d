"""The unpack rings of the int8-operand GEMM kernels, checked on the CPU: every interleaving of the packed-weight copies, the
two unpack groups and the MMAs is walked, with the ring sizes and the order of the two waits taken from the kernel sources.

The barriers are what the hardware gives: a wait names the parity of a phase, so a wait for phase n also passes while the
barrier is still in phase n - 1.  A group must never take a slot whose copy has not landed, and the producer must never arm a
slot that has not been given back."""
from __future__ import annotations

import os
import re

import pytest

from conftest import ROOT


def source(name: str) -> str:
    return open(os.path.join(ROOT, "quest_b200", "csrc", name)).read()


def full_p_first(text: str) -> bool:
    """Whether the unpack warps wait for the packed copy before they wait for their operand stage."""
    pairs = re.findall(r"ok = mbar_wait\((\w+) \+ 8 \* \w+, [^;]*?mbar_wait\((\w+) \+ 8 \* \w+, [^;]*;", text)
    pairs = [p for p in pairs if set(p) == {"full_p", "empty"}]
    assert len(pairs) == 1
    return pairs[0][0] == "full_p"


def wait_passes(completed: int, phase: int) -> bool:
    """try_wait.parity for the end of phase `phase` on a barrier that has ended `completed` phases."""
    return (completed & 1) != (phase & 1)


def find_fault(stages: int, p_stages: int, copy_first: bool, steps: int):
    """The first fault over all interleavings of `steps` K steps, or None.  State: copies issued, which of them have landed,
    what each group does (step, waits passed), steps whose MMAs have completed."""
    def uses_ended(done, slot, ring):  # uses of a ring slot for which done(step) holds
        return sum(1 for it in range(slot, steps, ring) if done(it))

    start = (0, 0, ((0, 0), (1, 0)), 0)
    seen, todo = {start}, [start]
    while todo:
        issued, landed, groups, mma = todo.pop()

        def unpacked(it):
            return groups[it & 1][0] > it

        nxt = []
        if issued < steps:  # producer: slot given back by its use before?
            use = issued // p_stages
            if wait_passes(uses_ended(unpacked, issued % p_stages, p_stages), use - 1) or use == 0:
                if use > 0 and not unpacked(issued - p_stages):
                    return f"copy of step {issued} is armed before step {issued - p_stages} is unpacked"
                nxt.append((issued + 1, landed, groups, mma))
        for it in range(issued):  # copies land in any order
            if not landed >> it & 1:
                nxt.append((issued, landed | 1 << it, groups, mma))
        for g, (it, passed) in enumerate(groups):
            if it >= steps:
                continue
            on_copy = (passed == 0) == copy_first
            if on_copy:
                ok = wait_passes(uses_ended(lambda j: landed >> j & 1, it % p_stages, p_stages), it // p_stages)
            else:
                ok = it < stages or wait_passes(uses_ended(lambda j: j < mma, it % stages, stages), it // stages - 1)
            if not ok:
                continue
            if passed == 0:
                new = (it, 1)
            else:
                if not landed >> it & 1:
                    return f"step {it} is unpacked before its copy has landed"
                if it >= stages and mma <= it - stages:
                    return f"step {it} overwrites operands that the MMAs of step {it - stages} still read"
                new = (it + 2, 0)
            nxt.append((issued, landed, (new, groups[1]) if g == 0 else (groups[0], new), mma))
        if mma < steps and unpacked(mma):
            nxt.append((issued, landed, groups, mma + 1))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


def test_the_model_sees_the_fault():
    """Two groups that take turns on an odd ring and wait for the copy first: nothing has ended the slot's use before."""
    assert "before its copy has landed" in find_fault(5, 5, True, 12)
    assert find_fault(5, 6, True, 12) is None and find_fault(3, 5, True, 12) is None
    assert find_fault(7, 5, False, 12) is not None  # more operand stages than packed slots, which the order does not cover


def test_pair_kernel_rings():
    text = source("gemm_i4_pair.cuh")
    stages, p_stages = (int(re.search(rf"constexpr int {name} = (\d+);", text).group(1)) for name in ("STAGES", "P_STAGES"))
    assert find_fault(stages, p_stages, full_p_first(text), 2 * p_stages + 4) is None


@pytest.mark.parametrize("tokens", [16, 32, 64, 128])
def test_few_token_kernel_rings(tokens):
    text = source("gemm_i4_skinny.cuh")

    def stages(name):  # the C expression of the constant, with TN = tokens
        expr = re.search(rf"constexpr int {name} = ([^;]+);", text).group(1)
        while "?" in expr:
            cond, rest = expr.split("?", 1)
            depth, i = 0, 0
            while depth or rest[i] != ":":
                depth += (rest[i] == "(") - (rest[i] == ")")
                i += 1
            taken = eval(cond.replace("||", " or ").replace("TN", str(tokens)))
            expr = (rest[:i] if taken else rest[i + 1:]).strip()
            if expr.startswith("(") and expr.endswith(")"):
                expr = expr[1:-1]
        return int(expr)

    u, p = stages("U_STAGES"), stages("P_STAGES")
    if p > 6:  # a slot of an even ring always belongs to the same group; six slots stand for it
        assert p % 2 == 0
        p = 6
    assert find_fault(u, p, full_p_first(text), 2 * p + 3) is None
