"""How the CTAs of a cluster leave when a bounded wait has run out, restated as a
schedule and run under random interleavings on the CPU: no CTA leaves while a
message (an asynchronous store into its shared memory) is still on its way to it,
and every wait on the way out ends. A cluster barrier alone does not give that: it
does not order asynchronous stores. Whether the kernels do more than the barrier,
and their ring depths, are read from their source.

The analysis (csrc/analysis.cu): CTA k sends MB m's decision to every CTA onto the
mbarrier m % ring, armed for one message a CTA; its helper takes the phases in
order, arming each again, and prepares MB m while m < taken + 2.

The split loop-filter pass (csrc/lf.cu): the CTA above sends column c's rows at
column c + 1, once column c - 2's are back; the CTA below takes them in at column c
and returns them, a share a lane. A lane whose wait runs out closes its end of the
link."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "oxideav-vp8_b200", "csrc")


def source(name):
    return open(os.path.join(CSRC, name)).read()


class Violation(Exception):
    pass


class Phases:
    """An mbarrier as the kernels use it: `armed` phases so far (each armed for
    `messages`), the messages landed or taken off in each."""

    def __init__(self, messages, armed):
        self.messages, self.armed, self.landed = messages, armed, {}

    def add(self, phase, n=1):
        self.landed[phase] = self.landed.get(phase, 0) + n
        assert self.landed[phase] <= self.messages

    def done(self, phase):
        return phase < self.armed and self.landed.get(phase, 0) == self.messages


def analysis(n_ctas, mbs, cols, seed, awaits, ring):
    rnd = random.Random(seed)
    stop_at = rnd.randrange(0, 40 * n_ctas) if rnd.random() < 0.9 else 10 ** 9
    bars = [[Phases(n_ctas, 1) for _ in range(ring)] for _ in range(n_ctas)]
    sent, pre, pub = [0] * n_ctas, [0] * n_ctas, [0] * n_ctas
    helper_in, search_in, stopped = [True] * n_ctas, [True] * n_ctas, [False] * n_ctas
    flying = []  # (to, mb)
    status, step = False, 0

    def done(k, m):
        return bars[k][m % ring].done(m // ring)

    while any(helper_in) or any(search_in):
        step += 1
        status = status or step >= stop_at
        assert step < 200000, "no end"
        act = rnd.randrange(3)
        k = rnd.randrange(n_ctas)
        if act == 0 and flying and rnd.random() < 0.7:
            to, m = flying.pop(rnd.randrange(len(flying)))
            assert bars[to][m % ring].armed == m // ring + 1, "a message ahead of its phase"
            bars[to][m % ring].add(m // ring)
        elif act == 1 and helper_in[k]:
            if pub[k] < mbs and done(k, pub[k]):
                bars[k][pub[k] % ring].armed += 1
                pub[k] += 1
            elif pre[k] < mbs and pre[k] < pub[k] + 2 and not status:
                pre[k] += 1
            elif pub[k] == mbs:
                helper_in[k] = False
            elif status:
                stopped[k], helper_in[k] = True, False
        elif act == 2 and search_in[k]:
            m = sent[k]
            if m == mbs:
                search_in[k] = False
            elif m < pre[k] and (m % cols == 0 or done(k, m - 1)):
                flying += [(to, m) for to in range(n_ctas)]
                sent[k] += 1
            elif stopped[k]:
                search_in[k] = False
    # The cluster barrier; then each CTA leaves on its own.
    inside = set(range(n_ctas))
    if awaits:
        for k in range(n_ctas):
            for m in range(pub[k], max(sent)):
                b = bars[k][m % ring]
                assert b.armed == m // ring + 1, "an unarmed phase is awaited"
                b.add(m // ring, sum(s <= m for s in sent))
    while inside:
        step += 1
        assert step < 400000, "a wait on the way out does not end"
        if flying and rnd.random() < 0.5:
            to, m = flying.pop(rnd.randrange(len(flying)))
            if to not in inside:
                raise Violation("a message arrived after its target had left")
            bars[to][m % ring].add(m // ring)
            continue
        k = rnd.choice(sorted(inside))
        if not awaits or all(done(k, m) for m in range(pub[k], max(sent))):
            inside.remove(k)
    if flying:
        raise Violation("a message was on its way when its target left")


def analysis_constants():
    text = source("analysis.cu")
    kernel = text[text.index("analysis_kernel(const __grid_constant__"):]
    leave = kernel[kernel.index("auto leave = ["):kernel.index("  };")]
    awaits = leave.index("cluster_sync();") < leave.index("await_decisions(")
    # Both ways out: stopping, and the end of the kernel.
    awaits = awaits and kernel.count("leave();") == 2 and "leave();\n}" in kernel and "leave();\n        return;" in kernel
    return awaits, int(re.search(r"DEC_RING = (\d+);", text).group(1))


@pytest.mark.parametrize("n_ctas", [1, 2, 3])
def test_analysis_ctas_leave_after_their_messages(n_ctas):
    awaits, ring = analysis_constants()
    for seed in range(400):
        analysis(n_ctas, 12, 5, seed, awaits, ring)


def test_a_barrier_alone_is_not_enough():
    with pytest.raises(Violation):
        for seed in range(400):
            analysis(2, 12, 5, seed, False, 4)


def split_pass(n_ctas, rows, cols, lanes, seed, awaits):
    """CTA k holds `rows` rows; row s of all runs column t - s at step t. A message is
    `lanes` shares, one a lane; lane 0 arms the phases."""
    rnd = random.Random(seed)
    patience = rnd.choice([0, 1, 3, 30])  # tries of a wait before it runs out
    pace = rnd.choice([0.4, 0.1, 0.02])  # of the messages' arrival
    depth = 3  # columns from an MB to the one that takes its slot
    ins = [[Phases(lanes, 1) for _ in range(2)] for _ in range(n_ctas)]
    rets = [[Phases(lanes, 1) for _ in range(2)] for _ in range(n_ctas)]
    n_in, n_back, n_down = ([[0] * lanes for _ in range(n_ctas)] for _ in range(3))
    given_up = [False] * n_ctas
    flying = []
    inside = set(range(n_ctas))

    def land():
        box, k, m = flying.pop(rnd.randrange(len(flying)))
        if k not in inside:
            raise Violation("a message arrived after its target had left")
        # A share may come before its phase is armed, not before the one in front is over.
        assert box[k][m & 1].armed >= m // 2 + 1 or box[k][m & 1].done(m // 2 - 1), "a message ahead of its phase"
        box[k][m & 1].add(m // 2)

    def waits(box, k, m):
        tries = 0
        while not box[k][m & 1].done(m // 2):
            tries += 1
            if tries > patience or given_up[k]:
                given_up[k] = True
                return False
            yield
        return True

    def lane(k, q):
        up, down = k > 0, k + 1 < n_ctas
        for t in range(n_ctas * rows + cols + depth):
            c = t - (k + 1) * rows + 1  # the last row's column
            if down and depth <= c < cols + depth:
                down = yield from waits(rets, k, c - depth)
                if down:
                    rets[k][c - depth & 1].armed += q == 0
                    n_back[k][q] += 1
            if down and 1 <= c <= cols:
                flying.append((ins, k + 1, c - 1))
                n_down[k][q] += 1
            yield "barrier"
            c = t - k * rows  # the first row's
            if up and 0 <= c < cols:
                up = yield from waits(ins, k, c)
                if up:
                    ins[k][c & 1].armed += q == 0
                    flying.append((rets, k - 1, c))
                    n_in[k][q] += 1
            yield "barrier"

    agents = {(k, q): lane(k, q) for k in range(n_ctas) for q in range(lanes)}
    held = set()
    while agents:
        if flying and rnd.random() < pace:
            land()
        a = rnd.choice(sorted(set(agents) - held))
        got = next(agents[a], "end")
        if got == "end":
            del agents[a]
        elif got == "barrier":
            held.add(a)
            if all((a[0], q) in held for q in range(lanes)):
                held -= {(a[0], q) for q in range(lanes)}
    owed = {k: [] for k in range(n_ctas)}
    for k in range(n_ctas):
        for box, got, sent in ((ins, n_in[k][0], n_down[k - 1] if k else [0]),
                               (rets, n_back[k][0], n_in[k + 1] if k + 1 < n_ctas else [0])):
            for m in range(got, max(sent)):
                assert box[k][m & 1].armed == m // 2 + 1, "an unarmed phase is awaited"
                if awaits:
                    box[k][m & 1].add(m // 2, sum(x <= m for x in sent))
                owed[k].append((box, m))
    step = 0
    while inside:
        step += 1
        assert step < 100000, "a wait on the way out does not end"
        if flying and rnd.random() < 0.5:
            land()
            continue
        k = rnd.choice(sorted(inside))
        if not awaits or all(box[k][m & 1].done(m // 2) for box, m in owed[k]):
            inside.remove(k)
    if flying:
        raise Violation("a message was on its way when its target left")
    return any(given_up)


def split_awaits():
    text = source("lf.cu")
    body = text[text.index("void leave_split("):text.index("void class_limits(")]
    return body.count("await_messages(") == 2 and body.index("barrier.cluster.wait") < body.index("await_messages(")


@pytest.mark.parametrize("n_ctas,rows,lanes", [(2, 1, 1), (2, 3, 2), (4, 1, 2), (3, 2, 4)])
def test_split_pass_ctas_leave_after_their_messages(n_ctas, rows, lanes):
    awaits = split_awaits()
    assert any([split_pass(n_ctas, rows, 7, lanes, seed, awaits) for seed in range(250)])


def test_a_barrier_alone_is_not_enough_for_a_split_pass():
    with pytest.raises(Violation):
        for seed in range(400):
            split_pass(4, 1, 7, 1, seed, False)
