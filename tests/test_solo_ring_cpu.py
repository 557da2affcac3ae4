"""The barriers of attn_solo_kernel, explored on the CPU: no MMA reads a K or V tile that has not landed.

A model of the producer, the issuer and the two softmax groups, in which loads land in any order and every interleaving is
walked.  An mbarrier parity wait for use ``u`` of a slot blocks only while exactly ``u`` uses are complete: with ``u - 1``
complete it returns at once, which is the trap.  The order of the group's waits is read from the kernel's source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diffusers-tpu_b200", "csrc", "attn_solo.cuh")


def _source():
    with open(SOURCE) as f:
        return f.read()


def _stages():
    return int(re.search(r"kSoloStages = (\d+);", _source()).group(1))


def _wait_order():
    """The waits of a softmax group for its tile e, in program order."""
    text = _source()
    loop = text[text.index("for (int j = 0; j < n_own"):]
    loop = loop[:loop.index("softmax_tile<")]
    names = {"s_full[t]": "S", "kv_full[iv": "V", "kv_full[ik": "K"}
    return [names[m.group(1)] for m in re.finditer(r"mbar_wait\(smem_u32\(&bars->(s_full\[t\]|kv_full\[iv|kv_full\[ik)", loop)]


def _explore(n, order, stages):
    """Every reachable state of a block of n key tiles: (an MMA read a tile that had not landed, all of them finish)."""
    def place_k(e):
        return 0 if e == 0 else 2 * e - 1

    def place_v(e):
        return 2 * n - 1 if e == n - 1 else 2 * e + 2

    def passes(complete, use):
        return (complete & 1) != (use & 1)

    # issuer program: wait for a load, wait for P(e), or use the tile at a place (which frees its slot) and publish S
    issuer = []
    for t in range(min(n, 2)):
        issuer += [("load", place_k(t)), ("use", place_k(t), t)]
    for e in range(n):
        issuer += [("P", e), ("use", place_v(e), None)]
        if e + 2 < n:
            issuer.append(("use", place_k(e + 2), e + 2))
    groups = []
    for t in range(2):
        program = []
        for e in range(t, n, 2):
            waits = {"S": ("S", e), "V": ("load", place_v(e)), "K": ("load", place_k(e + 2)) if e + 2 < n else None}
            program += [waits[w] for w in order if waits[w]] + [("publish", e)]
        groups.append(program)

    # state: loads requested, landed (bit set), issuer position, group positions
    start = (0, 0, 0, 0, 0)
    seen, stack, early, finished = {start}, [start], False, 0
    while stack:
        requested, landed, ipos, g0, g1 = state = stack.pop()

        def complete(slot):          # uses of the slot that have landed
            return sum(1 for i in range(slot, requested, stages) if landed >> i & 1)

        freed = {op[1] for op in issuer[:ipos] if op[0] == "use"}
        scores = {op[2] for op in issuer[:ipos] if op[0] == "use" and op[2] is not None}
        published = {op[1] for pos, prog in ((g0, groups[0]), (g1, groups[1])) for op in prog[:pos] if op[0] == "publish"}
        nxt = []
        if requested < 2 * n and (requested < stages or requested - stages in freed):
            nxt.append((requested + 1, landed, ipos, g0, g1))
        for i in range(requested):
            if not landed >> i & 1:
                nxt.append((requested, landed | 1 << i, ipos, g0, g1))
        if ipos < len(issuer):
            op = issuer[ipos]
            if op[0] == "use" and not landed >> op[1] & 1:
                early = True
                continue
            if op[0] == "use" or (op[0] == "P" and op[1] in published) or (
                    op[0] == "load" and passes(complete(op[1] % stages), op[1] // stages)):
                nxt.append((requested, landed, ipos + 1, g0, g1))
        for t, pos in enumerate((g0, g1)):
            if pos < len(groups[t]):
                op = groups[t][pos]
                if op[0] == "publish" or (op[0] == "S" and op[1] in scores) or (
                        op[0] == "load" and passes(complete(op[1] % stages), op[1] // stages)):
                    nxt.append((requested, landed, ipos, g0 + (t == 0), g1 + (t == 1)))
        if not nxt:
            finished += state == (2 * n, (1 << 2 * n) - 1, len(issuer), len(groups[0]), len(groups[1]))
            assert finished, f"stuck in {state}"
        for s in nxt:
            if s not in seen:
                seen.add(s)
                stack.append(s)
    return early, finished == 1


def test_the_model_is_of_the_kernel():
    text = _source()
    assert "place_k = [&](int e) { return e == 0 ? 0 : 2 * e - 1; };" in text
    assert "place_v = [&](int e) { return e == n_tiles - 1 ? 2 * n_tiles - 1 : 2 * e + 2; };" in text
    assert sorted(_wait_order()) == ["K", "S", "V"]


@pytest.mark.parametrize("n", range(1, 13))
def test_no_tile_is_read_before_it_has_landed(n):
    early, finished = _explore(n, _wait_order(), _stages())
    assert not early and finished


def test_the_model_sees_the_trap():
    """With the load checks in front of the wait for S, a check can pass one use of the slot too early."""
    assert [_explore(n, ["V", "K", "S"], 5)[0] for n in range(1, 7)] == [False, False, False, True, True, True]
