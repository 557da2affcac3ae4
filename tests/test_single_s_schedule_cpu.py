"""The barriers of the attention kernels, explored on the CPU, for both block forms.

A model of the producer, the two issuers and the two softmax groups, in which loads land in any order and every interleaving is
walked.  The one S buffer passes between the groups, each of which has a P of its own.  An mbarrier parity wait for phase
``u`` passes whenever the number of finished phases has the other parity than ``u``, so it can pass early or block for ever; the model
waits the same way and looks at each step for an MMA that reads a K or V tile that has not landed, overwrites an S that has
not been read, or reads a P that is not written, and for a P that is written while it is still to be read.  The places in
the ring and the load checks of a group are read from the kernels' sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "diffusers-tpu_b200", "csrc")
FORMS = {"pair": ("attn_kernel.cuh", r"kStages = (\d+);"), "solo": ("attn_solo.cuh", r"kSoloStages = (\d+);")}


def _source(form):
    with open(os.path.join(CSRC, FORMS[form][0])) as f:
        return f.read()


def _stages(form):
    return int(re.search(FORMS[form][1], _source(form)).group(1))


def place_k(e):
    return 0 if e == 0 else 2 * e - 1


def place_v(e, n):
    return 2 * n - 1 if e == n - 1 else 2 * e + 2


def _programs(form, n, checked=True):
    """Programs of the two issuers and the two groups for a block of n key tiles.  Step s is one S tile: key tile s // 2 of
    query tile s % 2 (pair) or key tile s (solo).  Without ``checked`` nothing waits for loads after the first."""
    tiles = (lambda s: s // 2) if form == "pair" else (lambda s: s)
    steps = 2 * n if form == "pair" else n

    def frees(s):                        # the last S tile of a key tile gives its K (and its P V its V) back
        return form == "solo" or s % 2 == 1

    scores, values = [], []
    for s in range(steps):
        if s == 0 or (checked and form == "pair" and s % 2 == 0):
            scores.append(("load", place_k(tiles(s))))
        if s > 0:
            scores.append(("s_free", s - 1))
        scores.append(("qk", s, place_k(tiles(s)), frees(s)))
        if checked and form == "pair" and s % 2 == 0:
            values.append(("load", place_v(tiles(s), n)))
        values += [("p", s), ("pv", s, place_v(tiles(s), n), frees(s))]
    groups = []
    for t in range(2):
        program = []
        for s in range(t, steps, 2):
            program.append(("s", s))
            if checked and form == "solo":
                program.append(("load", place_v(s, n)))
                if s + 1 < steps:
                    program.append(("load", place_k(s + 1)))
            program.append(("read", s))
            if s >= 2:
                program.append(("pv_done", s - 2))
            program.append(("write", s))
        if program:
            program.append(("pv_done", s))
        groups.append(program)
    return scores, values, groups[0], groups[1]


def _explore(form, n, stages, checked=True):
    """Every reachable state: what went wrong first, or None when all interleavings finish."""
    programs = _programs(form, n, checked)
    freed_by = {op[2]: (i, k) for i in (0, 1) for k, op in enumerate(programs[i]) if op[0] in ("qk", "pv") and op[3]}
    loads = 2 * n
    start = (0, 0, (0, 0, 0, 0))         # loads asked for, loads landed (bits), positions in the programs
    seen, stack, finished = {start}, [start], False

    def passes(done, phase):             # a parity wait for `phase` (0-based) with `done` phases finished
        return (done & 1) != (phase & 1)

    while stack:
        requested, landed, at = state = stack.pop()

        def count(kind, t):              # phases of query tile or parity t that are finished
            i = {"qk": 0, "pv": 1}.get(kind, 2 + t)
            return sum(1 for op in programs[i][:at[i]] if op[0] == kind and op[1] % 2 == t)

        def ready(op):
            kind, s = op[0], op[1]
            if kind == "load":
                slot = s % stages
                return passes(sum(1 for i in range(slot, requested, stages) if landed >> i & 1), s // stages)
            if kind == "s_free":
                return passes(count("read", 0) + count("read", 1), s)
            done = {"p": "write", "s": "qk", "pv_done": "pv"}.get(kind)
            return done is None or passes(count(done, s % 2), s // 2)

        nxt = []
        if requested < loads:
            freeing = freed_by.get(requested - stages)
            if freeing is None or at[freeing[0]] > freeing[1]:
                nxt.append((requested + 1, landed, at))
        for i in range(requested):
            if not landed >> i & 1:
                nxt.append((requested, landed | 1 << i, at))
        for i in range(4):
            if at[i] == len(programs[i]) or not ready(programs[i][at[i]]):
                continue
            op = programs[i][at[i]]
            kind, s = op[0], op[1]
            if kind in ("qk", "pv") and not landed >> op[2] & 1:
                return f"{op} reads a tile that has not landed"
            if kind == "qk" and count("read", 0) + count("read", 1) != s:
                return f"{op} overwrites S"
            if kind == "pv" and count("write", s % 2) != s // 2 + 1:
                return f"{op} reads P"
            if kind == "read" and count("qk", s % 2) != s // 2 + 1:
                return f"{op}: S is not there"
            if kind == "write" and count("pv", s % 2) != s // 2:
                return f"{op} overwrites P"
            nxt.append((requested, landed, at[:i] + (at[i] + 1,) + at[i + 1:]))
        if not nxt:
            if state != (loads, (1 << loads) - 1, tuple(len(p) for p in programs)):
                return f"stuck in {state}"
            finished = True
        for s in nxt:
            if s not in seen:
                seen.add(s)
                stack.append(s)
    return None if finished else "never finished"


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("n", range(1, 9))
def test_every_interleaving_is_ordered_and_ends(form, n):
    assert _explore(form, n, _stages(form)) is None


@pytest.mark.parametrize("form", FORMS)
def test_the_model_is_of_the_kernel(form):
    text = _source(form)
    assert "place_k = [&](int e) { return e == 0 ? 0 : 2 * e - 1; };" in text
    assert "place_v = [&](int e) { return e == n_tiles - 1 ? 2 * n_tiles - 1 : 2 * e + 2; };" in text
    group = text[text.index("// ------------------------------------------------------------------ softmax groups"):]
    issuers = text[text.index("// ------------------------------------------------------------------ issuer of S"):text.index(group)]
    checks = issuers if form == "pair" else group[group.index("bars->s_full[t]"):group.index("softmax_tile<")]
    assert all(re.search(w, checks) for w in (("place_k\\(j\\)", "place_v\\(j\\)") if form == "pair" else ("place_k\\(e \\+ 1\\)", "place_v\\(e\\)")))


@pytest.mark.parametrize("form", FORMS)
def test_the_model_sees_a_missing_check(form):
    assert "has not landed" in _explore(form, 4, _stages(form), checked=False)
