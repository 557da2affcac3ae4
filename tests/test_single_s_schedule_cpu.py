"""The barriers of the attention kernels, explored on the CPU, for all block forms.

The kernels' own sources are compiled for the host against ``host_trace/ptx.cuh``, which stands in for ``csrc/ptx.cuh`` and prints what a
thread waits for, arrives on, loads, issues and touches.  The printed programs of the producer, the two issuers and two warps
of each softmax group are then run against each other in every interleaving: loads land in any order, MMAs and commits run in
the order of their issuer at any time after it has issued them.  An mbarrier is its phase parity, the arrivals that the phase
still waits for and its outstanding bytes, so a parity wait can pass one use early or block for ever as the real one does.

One run of the programs says which write each access to S, P, O, Q, a slot of the K/V ring or the exchanged row statistics
follows, and that the accumulators come out as the sums over the right tiles; every other interleaving has to agree, and at the
end of a block nothing may still be in flight to its shared memory.  Small mistakes planted in a copy of the sources, one at
a time, have to be found.

Not covered: the 128 threads of a group are two, warps run one instruction stream (no divergence), waits do not run out."""
import functools
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "diffusers-tpu_b200", "csrc")
PANEL, TILE = 16384, 32768              # bytes of a 64-column panel and of a 128-row tile in shared memory


class Wrong(Exception):
    pass


# ---------------------------------------------------------------------------------------------------------------- programs
@pytest.fixture(scope="module")
def built(tmp_path_factory):
    """edit -> path of the tracing program, with the edit ((file, old, new, ...) or None) made in a copy of the sources."""
    @functools.cache
    def build(edit=None):
        folder = tmp_path_factory.mktemp("trace")
        for path in (os.path.join(HERE, "host_trace", "ptx.cuh"), os.path.join(HERE, "host_trace", "trace.cc"),
                     os.path.join(CSRC, "attn_kernel.cuh"), os.path.join(CSRC, "attn_solo.cuh")):
            with open(path) as f:
                text = f.read()
            if edit and os.path.basename(path) == edit[0]:
                for old, new in zip(edit[1::2], edit[2::2]):
                    assert text.count(old) == 1, f"{old!r} stands {text.count(old)} times in {edit[0]}"
                    text = text.replace(old, new)
            with open(folder / os.path.basename(path), "w") as f:
                f.write(text)
        subprocess.run(["g++", "-std=c++17", "-O0", "-w", "-I", str(folder), str(folder / "trace.cc"), "-o", str(folder / "trace")],
                       check=True, capture_output=True, text=True)
        return str(folder / "trace")

    return build


def _trace(program, form, n, mode, state):
    """role -> events between the block's first and last barrier, and barrier -> (name, arrivals per phase)."""
    text = subprocess.run([program, form, str(n), mode, state], check=True, capture_output=True, text=True).stdout
    roles, names, counts, events = {}, {}, {}, None
    for line in text.splitlines():
        kind, *args = line.split()
        if kind == "thread":
            events = roles[args[0]] = []
        elif kind == "name":
            names[int(args[0])] = args[1]
        elif kind == "init":
            counts[int(args[0])] = int(args[1])
        else:
            events.append((kind, *(int(a) if a.lstrip("-").isdigit() else a for a in args)))
    for role, events in roles.items():
        syncs = [i for i, e in enumerate(events) if e[0] == "sync"]
        assert len(syncs) == 2 and {e[0] for e in events[:syncs[0]]} <= {"before"}, role
        roles[role] = events[syncs[0] + 1:syncs[1]]
    assert set(names) == set(counts) and set(counts.values()) == {1, 128}
    return roles, names, counts


def _check_fences(role, events):
    """tcgen05 accesses of a thread stand behind a fence after a wait and in front of one before an arrival, stores complete."""
    fenced, pending, stored = True, False, False
    for kind, *_ in events:
        if kind == "wait":
            fenced = False
        elif kind == "after":
            fenced = True
        elif kind in ("ld", "st", "qk", "pv"):
            if not fenced:
                raise Wrong(f"{role}: {kind} behind a wait without a fence")
            pending, stored = kind in ("ld", "st"), stored or kind == "st"
        elif kind == "wait_st":
            stored = False
        elif kind == "before":
            pending = False
        elif kind == "arrive":
            if pending or stored:
                raise Wrong(f"{role}: arrival without a fence, or ahead of its stores")


def _programs(roles, form, warps):
    """The events as programs.  A program is a list of ("issue", bar to wait for or None, parity, operations issued after it), for the producer and
    the issuers, or of ("wait", bar, parity) and ("do", accesses, bar to arrive on or None), for a warp of a group; the loads and the two
    pipes are lists of (accesses, bar or None, bytes).  An access is (place, what, details)."""
    produce, loads, open_load = [], [], None
    for kind, *a in roles["load"]:
        if kind == "wait":
            produce.append(("wait", *a))
        elif kind == "expect":
            assert open_load is None
            open_load, size = [a[0], a[1], None], a[1]
        elif kind == "load":
            dst, source, bar, c0, row = a
            assert bar == open_load[0] and dst % TILE == c0 // 64 * PANEL and open_load[2] in (None, (dst // TILE, source, row))
            open_load[1:] = open_load[1] - PANEL, (dst // TILE, source, row)
            if open_load[1] == 0:
                parts = [(dst // TILE, w) for w in range(warps)] if source == "Q" else [dst // TILE]
                loads.append(([(part, "load", (source, row)) for part in parts], bar, size))
                produce.append(("push", len(loads)))
                open_load = None
    assert open_load is None

    def issuer(role, kind_of, width, accesses_of):
        program, pipe, batch = [], [], []
        for kind, *a in roles[role]:
            if kind == kind_of:
                batch.append(a)
                if len(batch) == width:
                    pipe.append((accesses_of(batch), None, 0))
                    program.append(("push", len(pipe)))
                    batch = []
            elif kind in ("wait", "commit"):
                assert not batch
                if kind == "commit":
                    pipe.append(([], a[0], 0))
                program.append(("push", len(pipe)) if kind == "commit" else ("wait", *a))
        assert not batch
        return program, pipe

    def scores(batch):                  # a whole tile of Q times a whole tile of K over all of S
        q, k = batch[0][1] // TILE, batch[0][2] // TILE
        offsets = [i % 4 * 32 + i // 4 * PANEL for i in range(len(batch))]
        assert batch == [[0, q * TILE + o, k * TILE + o, int(i > 0)] for i, o in enumerate(offsets)]
        return [((q, w), "read", None) for w in range(warps)] + [(k, "read", None), ("S", "scores", ((q, 0), k))]

    def values(batch):                  # 64 keys of P times those rows of V, into or onto all of O
        t, v = (batch[0][0] - 256) // 128, batch[0][2] // TILE
        half = (batch[0][1] - 128 - 64 * t) // 32
        assert batch == [[256 + 128 * t, 128 + 64 * t + 32 * half + 8 * i, v * TILE + (4 * half + i) * 2048, int(i > 0 or batch[0][3])]
                         for i in range(4)]
        probs = [("P", t, 2 * half + c, w) for c in range(2) for w in range(warps)]
        return [(v, "read", None)] + [(p, "read", None) for p in probs] + [
            (("O", t, c, w), "values", (probs, v, half, batch[0][3])) for c in range(4) for w in range(warps)]

    score_program, score_pipe = issuer("scores", "qk", 4 if form.endswith("8") else 8, scores)
    value_program, value_pipe = issuer("values", "pv", 4, values)
    groups = []
    for t in range(2):
        for w in range(warps):
            role, program, todo = (t, w), [], []
            for kind, *a in roles[f"group{t}.{w}"]:
                if kind in ("wait", "arrive"):
                    if todo or kind == "arrive":
                        program.append(("do", todo, a[0] if kind == "arrive" else None))
                    todo = []
                    if kind == "wait":
                        program.append(("wait", *a))
                elif kind in ("ld", "st") and a[0] >= 256:
                    assert a[1] == 32
                    todo.append((("O", a[0] // 128 - 2, a[0] % 128 // 32, w), "read" if kind == "ld" else "rescale", role))
                elif kind == "ld":
                    assert a == [0, 128]
                    todo.append(("S", "read", role))
                elif kind == "st":
                    assert a[1] == 16
                    todo.append((("P", a[0] // 64 - 2, a[0] % 64 // 16, w), "probs", role))
                elif kind == "stage":      # a quarter of a Q tile takes the output rows of a warp
                    assert a[0] % TILE // (TILE // 4) == w
                    if not todo or todo[-1][1] != "stage":
                        todo.append(((a[0] // TILE, w), "stage", None))
                elif kind in ("put", "get"):
                    todo.append((("ml", w), "put" if kind == "put" else "read", None))
            groups.append(program + [("do", todo, None)])
    # What is issued behind a wait, or behind what is issued already, only enables the pipe: it needs no step of its own.
    issuers = []
    for program in (produce, score_program, value_program):
        merged, issued = [], 0
        for op in program:
            if op[0] == "wait":
                merged.append([op[1], op[2], issued])
            else:
                issued = op[1]
                if not merged:
                    merged.append([None, 0, 0])
                merged[-1][2] = issued
        issuers.append([("issue", *op) for op in merged])
    return issuers + groups, [loads, score_pipe, value_pipe]


# ------------------------------------------------------------------------------------------------------------------ execution
class Block:
    """The programs with places, barriers and operations as numbers, and their execution step by step.

    A state is (positions of the programs, positions of the two MMA pipes, loads in flight, barriers, last write of each place); a
    barrier is (parity of finished phases, arrivals that the phase waits for, bytes that it waits for)."""

    def __init__(self, programs, pipes, names, counts, warps):
        self.programs, self.pipes, self.names = programs, pipes, names
        self.bars = {b: i for i, b in enumerate(sorted(counts))}
        self.arrivals = [1 if counts[b] == 1 else warps for b in sorted(counts)]
        self.places = {}
        for accesses in [op[1] for p in programs for op in p if op[0] == "do"] + [op[0] for pipe in pipes for op in pipe]:
            for place, *_ in accesses:
                self.places.setdefault(place, len(self.places))
        self.ids = {}                    # number of a write
        self.follows = {}                # access -> number of the write that it follows, from the first run
        self.values, self.seen, self.result = {}, {}, {}
        self.start = ((0,) * len(programs), (0, 0), (), tuple((0, c, 0) for c in self.arrivals), (0,) * len(self.places))

    def name(self, bar):
        return self.names[bar]

    def arrive(self, bars, bar, count=1, size=0):
        i = self.bars[bar]
        parity, pending, tx = bars[i]
        pending, tx = pending - count, tx + size
        if pending < 0:
            raise Wrong(f"{self.name(bar)}: an arrival too many")
        if pending == 0 and tx == 0:
            parity, pending = parity ^ 1, self.arrivals[i]
        return bars[:i] + ((parity, pending, tx),) + bars[i + 1:]

    def touch(self, writes, accesses, op, learn):
        for n, (place, what, details) in enumerate(accesses):
            i, me = self.places[place], (op, n)
            if learn:
                self.follows[me] = writes[i]
                self.meaning(place, what, details)
            elif writes[i] != self.follows[me]:
                raise Wrong(f"{what} of {place} at the wrong time")
            if what != "read":
                writes = writes[:i] + (self.ids.setdefault(me, len(self.ids) + 1),) + writes[i + 1:]
        return writes

    def meaning(self, place, what, details):
        """What the access does to what stands there, in terms of tiles."""
        v = self.values
        if what == "load":
            v[place] = details
        elif what == "scores":
            v[place] = (v.get(details[0]), v.get(details[1]))
        elif what == "read" and details is not None:
            if place == "S":
                self.seen[details] = v.get("S")
            else:
                self.seen[details, place] = self.result[details, place] = v.get(place)
        elif what == "probs":
            v[place] = self.seen.get(details)
        elif what == "rescale":          # without a read before it, a carried state comes in
            v[place] = self.seen.get((details, place), ("carried",))
        elif what == "values":
            probs, tile, half, onto = details
            if len({v.get(p) for p in probs}) != 1:
                raise Wrong("P of two tiles")
            v[place] = (v.get(place) or ("nothing",) if onto else ()) + ((v.get(probs[0]), v.get(tile), half),)

    def steps(self, state, learn=False):
        """The states after each step that can be taken."""
        at, pipe_at, flying, bars, writes = state
        for i, program in enumerate(self.programs):
            if at[i] == len(program):
                continue
            op, after = program[at[i]], at[:i] + (at[i] + 1,) + at[i + 1:]
            if op[0] != "do" and op[1] is not None and bars[self.bars[op[1]]][0] == op[2]:
                continue
            if op[0] == "do":
                w = self.touch(writes, op[1], (i, at[i]), learn)
                yield after, pipe_at, flying, self.arrive(bars, op[2]) if op[2] is not None else bars, w
            elif i == 0:                 # expect_tx, and the loads are on their way
                first, now = program[at[0] - 1][3] if at[0] else 0, bars
                for load in range(first, op[3]):
                    now = self.arrive(now, self.pipes[0][load][1], 1, self.pipes[0][load][2])
                yield after, pipe_at, flying + tuple(range(first, op[3])), now, writes
            else:
                yield after, pipe_at, flying, bars, writes
        for k in range(2):
            if at[k + 1] and pipe_at[k] < self.programs[k + 1][at[k + 1] - 1][3]:
                accesses, bar, _ = self.pipes[k + 1][pipe_at[k]]
                w = self.touch(writes, accesses, ("pipe", k, pipe_at[k]), learn)
                after = (pipe_at[0] + (k == 0), pipe_at[1] + (k == 1))
                yield at, after, flying, self.arrive(bars, bar) if bar is not None else bars, w
        for n, load in enumerate(flying):
            accesses, bar, size = self.pipes[0][load]
            w = self.touch(writes, accesses, ("load", load), learn)
            yield at, pipe_at, flying[:n] + flying[n + 1:], self.arrive(bars, bar, 0, -size), w

    def ended(self, state):
        return all(a == len(p) for a, p in zip(state[0], self.programs))

    def in_flight(self, state):
        return bool(state[2]) or state[1] != tuple(len(p) for p in self.pipes[1:])

    def first_run(self):
        state = self.start
        while not (self.ended(state) and not self.in_flight(state)):
            state = next(self.steps(state, learn=True), None)
            if state is None:
                raise Wrong("stuck")

    def explore(self):
        """Walks every interleaving; the number of states."""
        seen, stack = {self.start}, [self.start]
        while stack:
            state = stack.pop()
            if self.ended(state):
                if self.in_flight(state):
                    raise Wrong("in flight at the end of the block")
                continue
            moved = False
            for after in self.steps(state):
                moved = True
                if after not in seen:
                    seen.add(after)
                    stack.append(after)
            if not moved:
                waits = [self.name(p[a][1]) for p, a in zip(self.programs, state[0]) if a < len(p) and p[a][0] != "do"]
                raise Wrong(f"stuck, waiting for {waits}")
        return len(seen)


def _run(program, form, n, mode="steady", state="fresh", warps=1):
    """What goes wrong in some interleaving of a block of n key tiles, or None."""
    roles, names, counts = _trace(program, form, n, mode, state)
    try:
        for role, events in roles.items():
            _check_fences(role, events)
        block = Block(*_programs(roles, form, warps), names, counts, warps)
        block.first_run()
        # every accumulator that leaves the block: P of the group's key tiles times V of the same, in order, from the right Q and K
        solo, base = form.startswith("solo"), 256 if form == "pieces" else 0
        for t in range(2):
            tiles = range(t, n, 2) if solo else range(n)
            carried = state == "carried" and (t == 0 or not solo)
            want = ("carried",) if carried else ()
            for e in tiles:
                s = (("Q", 0 if solo else 128 * t), ("K", base + 128 * e))
                want += ((s, ("V", base + 128 * e), 0), (s, ("V", base + 128 * e), 1))
            for w in range(warps):
                for c in range(4):
                    place = ("O", t, c, w)
                    reader = (0 if solo else t, w)
                    if tiles and (block.result.get((reader, place)) != want or block.values.get(place) != want):
                        raise Wrong(f"{place} is not the sum over its tiles")
        block.explore()
    except Wrong as e:
        return str(e)
    return None


# ------------------------------------------------------------------------------------------------------------------------ tests
@pytest.mark.parametrize("form", ["pair", "solo"])
@pytest.mark.parametrize("n", range(1, 9))
def test_every_interleaving_is_ordered_and_ends(built, form, n):
    assert _run(built(), form, n) is None


@pytest.mark.parametrize("form", ["pair", "pair8", "pieces", "solo", "solo8"])
@pytest.mark.parametrize("mode,state,n,warps", [
    ("growing", "fresh", 5, 1), ("growing", "fresh", 2, 2), ("bounded", "fresh", 4, 1), ("steady", "fresh", 2, 2),
    ("steady", "carried", 3, 1), ("growing", "carried", 3, 1), ("bounded", "carried", 2, 2), ("growing", "carried", 1, 2),
])
def test_every_form_and_softmax_is_ordered_and_ends(built, form, mode, state, n, warps):
    """Offsets that move at every tile (O is rescaled), bounded logits, a running state; two warps of a group out of step."""
    if form == "pieces" and state == "carried":
        state = "fresh"                 # a piece starts its own state
    assert _run(built(), form, n, mode, state, warps) is None


@pytest.mark.parametrize("form", ["pair", "pair8", "pieces", "solo", "solo8"])
@pytest.mark.parametrize("mode", ["growing", "bounded"])
def test_nothing_stands_between_s_and_its_read(built, form, mode):
    """A group that has seen its S gives it back before it waits for anything else: the next Q K^T depends on that."""
    roles, names, _ = _trace(built(), form, 6, mode, "fresh")
    for role in [r for r in roles if r.startswith("group")]:
        order = [names[e[1]] for e in roles[role] if e[0] in ("wait", "arrive")]
        assert all(after == "s_free" for before, after in zip(order, order[1:]) if before == "s_full"), role


PAIR, SOLO = "attn_kernel.cuh", "attn_solo.cuh"
MISTAKES = {
    # Q K^T of the two-tile kernel
    "pair: S overwritten before it is read": ("pair", PAIR, "(j > 0 || t > 0)) ok = warp_wait(&bars->s_free, (t + 1) & 1, ctx, SITE_S_FREE)", "(j > 0 || t > 0)) ok = true"),
    "pair: parity of s_free": ("pair", PAIR, "&bars->s_free, (t + 1) & 1", "&bars->s_free, t & 1"),
    "pair: K not waited for": ("pair", PAIR, "const int i = place_k(j), slot = i % kStages;\n      for (int t = 0; t < kQTiles && ok; ++t) {\n        if (j == 0) ok = warp_wait(&bars->q_full[t], 0, ctx, SITE_Q_FULL + t);\n        if (ok && t == 0)", "const int i = place_k(j), slot = i % kStages;\n      for (int t = 0; t < kQTiles && ok; ++t) {\n        if (j == 0) ok = warp_wait(&bars->q_full[t], 0, ctx, SITE_Q_FULL + t);\n        if (false)"),
    "pair: Q not waited for": ("pair", PAIR, "if (j == 0) ok = warp_wait(&bars->q_full[t], 0", "if (j == 0) ok = t == 1 || warp_wait(&bars->q_full[t], 0"),
    "pair: K given back a query tile early": ("pair", PAIR, "issue_qk(t, slot);\n        if (t == kQTiles - 1", "issue_qk(t, slot);\n        if (t == 0"),
    "pair: arrivals that nobody waits for": ("pair", PAIR, "return i + kStages < 2 * n_tiles;", "return true;"),
    "pair: a slot that is reloaded is not given back": ("pair", PAIR, "return i + kStages < 2 * n_tiles;", "return i + kStages + 1 < 2 * n_tiles;"),
    # P V of the two-tile kernel
    "pair: V not waited for": ("pair", PAIR, "const int i = place_v(j), slot = i % kStages;\n      for (int t = 0; t < kQTiles && ok; ++t) {\n        if (t == 0)", "const int i = place_v(j), slot = i % kStages;\n      for (int t = 0; t < kQTiles && ok; ++t) {\n        if (false)"),
    "pair: first half of P not waited for": ("pair", PAIR, "if (ok) ok = warp_wait(&bars->p_lo[t], j & 1, ctx, SITE_P_FULL + t);", ""),
    "pair: second half of P not waited for": ("pair", PAIR, "ok = warp_wait(&bars->p_hi[t], j & 1, ctx, SITE_P_HI + t);", ""),
    "pair: parity of p_hi": ("pair", PAIR, "&bars->p_hi[t], j & 1", "&bars->p_hi[t], (j + 1) & 1"),
    "pair: V given back a query tile early": ("pair", PAIR, "commit_to(&bars->pv_done[t]);\n        if (t == kQTiles - 1", "commit_to(&bars->pv_done[t]);\n        if (t == 0"),
    "pair: the first P V adds to what was there": ("pair", PAIR, "issue_pv(t, slot, 0, j > 0 || o_preloaded);", "issue_pv(t, slot, 0, true);"),
    # the producer and the groups of the two-tile kernel
    "pair: slot reloaded before it is free": ("pair", PAIR, "if (use > 0) ok = mbar_wait(smem_u32(&bars->kv_empty[slot]), (use - 1) & 1, ctx, SITE_KV_EMPTY + slot);", ""),
    "pair: P written before the last P V": ("pair", PAIR, "if (j == 0) return true;", "return true;"),
    "pair: parity of pv_done": ("pair", PAIR, "&bars->pv_done[t], (j - 1) & 1", "&bars->pv_done[t], j & 1"),
    "pair: O read before the last P V": ("pair", PAIR, "if (ok) ok = warp_wait(&bars->pv_done[t], (n_tiles - 1) & 1, ctx, SITE_O_FULL + t);", ""),
    "softmax: S given back before it is read": ("pair", PAIR, "  tmem_ld128_sync(s_tmem, sr);\n  tc_fence_before();\n  mbar_arrive(bar_s_free);", "  tc_fence_before();\n  mbar_arrive(bar_s_free);\n  tmem_ld128_sync(s_tmem, sr);\n  tc_fence_before();"),
    "softmax: no fence between the read of S and giving it back": ("pair", PAIR, "  tmem_ld128_sync(s_tmem, sr);\n  tc_fence_before();\n", "  tmem_ld128_sync(s_tmem, sr);\n"),
    "pair: no fence behind the wait for the last P V": ("pair", PAIR, "ctx, SITE_O_FULL + t);\n    if (ok) {\n      tc_fence_after();", "ctx, SITE_O_FULL + t);\n    if (ok) {"),
    "softmax: P published before it is written": ("pair", PAIR, "    tmem_st16(p_tmem + half * 32 + 16, pk + 16);\n    tmem_wait_st();\n    tc_fence_before();\n    mbar_arrive(half == 0 ? bar_p_lo : bar_p_hi);", "    tc_fence_before();\n    mbar_arrive(half == 0 ? bar_p_lo : bar_p_hi);\n    tmem_st16(p_tmem + half * 32 + 16, pk + 16);\n    tmem_wait_st();\n    tc_fence_before();"),
    # the one-tile kernel
    "solo: arrivals that nobody waits for": ("solo", SOLO, "return i + kSoloStages < 2 * n_tiles;", "return true;"),
    "solo: S overwritten before it is read": ("solo", SOLO, "if (ok && e > 0) ok = warp_wait(&bars->s_free, (e - 1) & 1, ctx, SITE_S_FREE);", ""),
    "solo: V not waited for": ("solo", SOLO, "ok = warp_wait(&bars->kv_full[slot], (i / kSoloStages) & 1, ctx, SITE_KV_FULL + slot);\n      if (ok) ok = warp_wait(&bars->p_lo", "if (ok) ok = warp_wait(&bars->p_lo"),
    "solo: K not waited for": ("solo", SOLO, "ok = warp_wait(&bars->kv_full[slot], (i / kSoloStages) & 1, ctx, SITE_KV_FULL + slot);\n      if (ok && e > 0)", "if (ok && e > 0)"),
    "solo: first half of P not waited for": ("solo", SOLO, "if (ok) ok = warp_wait(&bars->p_lo[t], j & 1, ctx, SITE_P_FULL + t);", ""),
    "solo: second half of P not waited for": ("solo", SOLO, "ok = warp_wait(&bars->p_hi[t], j & 1, ctx, SITE_P_HI + t);", ""),
    "solo: P written before the last P V": ("solo", SOLO, "if (j == 0) return true;", "return true;"),
    "solo: slot reloaded before it is free": ("solo", SOLO, "if (use > 0) ok = mbar_wait(smem_u32(&bars->kv_empty[slot]), (use - 1) & 1, ctx, SITE_KV_EMPTY + slot);", ""),
    "solo: O read before the last P V": ("solo", SOLO, "if (ok && n_own > 0) ok = warp_wait(&bars->pv_done[t], (n_own - 1) & 1, ctx, SITE_O_FULL + t);", ""),
    "solo: statistics read before they are there": ("solo", SOLO, "ok = warp_wait(&bars->solo_ready, 0, ctx, kSiteSoloReady) && ", "ok = "),
}


@pytest.mark.parametrize("mistake", MISTAKES)
def test_a_planted_mistake_is_found(built, mistake):
    form, *edit = MISTAKES[mistake]
    assert any(_run(built(tuple(edit)), form, n, "growing") for n in (4, 5))
