"""How the CTAs of a cluster leave when a bounded wait has run out, restated as a
schedule and run under random interleavings on the CPU: no CTA leaves while a
message (an asynchronous store into its shared memory) is still on its way to it,
and every wait on the way out ends. A cluster barrier alone does not give that: it
does not order asynchronous stores. Whether the kernels do more than the barrier,
and their ring depths, are read from their source.

The analysis (csrc/analysis.cu): CTA k sends MB m's decision to every CTA onto the
mbarrier m % ring, armed for one message a CTA; its helper takes the phases in
order, arming each again, and prepares MB m while m < taken + 2."""
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
    barrier = kernel.rindex("cl.sync();", 0, kernel.index("kDefaultMvContexts"))
    tail = kernel[barrier:kernel.index("kDefaultMvContexts")]
    return "await_decisions(" in tail, int(re.search(r"DEC_RING = (\d+);", text).group(1))


@pytest.mark.parametrize("n_ctas", [1, 2, 3])
def test_analysis_ctas_leave_after_their_messages(n_ctas):
    awaits, ring = analysis_constants()
    for seed in range(400):
        analysis(n_ctas, 12, 5, seed, awaits, ring)


def test_a_barrier_alone_is_not_enough():
    with pytest.raises(Violation):
        for seed in range(400):
            analysis(2, 12, 5, seed, False, 4)
