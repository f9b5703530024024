"""The fused proposal net's hand-overs (lp_net_kernel in csrc/learned.cu), restated as
a schedule of its warps' roles and run under random interleavings on the CPU: no role
deadlocks, no parity wait (mbarrier.try_wait.parity) sees its barrier a phase further
than its parity can tell apart, no tile's matrix instructions read what is not
written yet or overwritten already, and no accumulator is taken before it is read.

The roles: ISSUERS warps that issue the tiles t = i, i + ISSUERS, ... of the 4 x 9 of
each map; two epilogue groups of which each reads back every other tile of a layer and
stores it; an output group that repacks a map's input, and makes the map's logits and
cells while the others are at the next map. Two meetings a map (a named barrier) join
the epilogue and output groups: before layer 2 is stored over layer 4's z, and once z
is complete. The constants are read from the kernel source."""
import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "oxideav-vp8_b200", "csrc", "learned.cu")
TEXT = open(SRC).read()
NS = TEXT[TEXT.index("namespace lpnet {"):TEXT.index("}  // namespace lpnet")]


def const(name):
    return int(re.search(rf"constexpr int {name} = (\d+);", NS).group(1))


TILES, NSLOT, ISSUERS, EPI, GRP = (const(k) for k in ("TILES", "NSLOT", "ISSUERS", "EPI", "GRP"))
GROUPS = EPI // GRP
PER_MAP = 4 * TILES


class Wrong(Exception):
    pass


class Net:
    """The two activation buffers as the tiles see them: who wrote each tile last."""

    def __init__(self):
        self.first = None  # B's first group: (map) whose input it holds
        self.b = {}        # B's other groups by tile: ("layer2", map) | ("z", map)
        self.a = {}        # A by tile: (layer, map)
        self.stage = None  # the bulk copy's map
        self.slots = {}    # accumulator -> (map, tile) in it, until read


def need(ok, what):
    if not ok:
        raise Wrong(what)


def slot(j, t):
    seq = PER_MAP * j + t
    return seq % NSLOT, seq // NSLOT


def around(u):
    return [w for w in (u - 1, u, u + 1) if 0 <= w < TILES]


def issuer(net, i, maps, issuers):
    def copy(j):
        need(net.stage is None, "a copy over an input that is not repacked")
        net.stage = j

    if i == 0:
        copy(0)
        yield ("arrive", "stage")
    for j in range(maps):
        yield ("wait", "input", j)
        if i == 0 and j + 1 < maps:
            copy(j + 1)
            yield ("arrive", "stage")
        for t in range(i, PER_MAP, issuers):
            layer, u = divmod(t, TILES)
            if layer > 0:
                for w in around(u):
                    yield ("wait", f"stored{layer - 1}_{w}", j)
            s, use = slot(j, t)
            if use > 0:
                yield ("wait", f"empty{s}", use - 1)
            need(s not in net.slots, "an accumulator taken before it is read")
            # The matrix instructions read their operands between issue and commit.
            for _ in range(2):
                if layer == 0:
                    need(net.first == j, "layer 1 reads another map's input")
                elif layer == 1:
                    need(all(net.a.get(w) == (0, j) for w in around(u)), "layer 2 reads A")
                elif layer == 2:
                    need(all(net.b.get(w) == ("layer2", j) for w in around(u)), "layer 3 reads B")
                else:
                    need(net.a.get(u) == (2, j), "layer 4 reads A")
                yield ("go",)
            net.slots[s] = (j, t)
            yield ("arrive", f"full{s}")


def epilogue(net, g, maps):
    def read(j, t):
        s, use = slot(j, t)
        yield ("wait", f"full{s}", use)
        need(net.slots.pop(s, None) == (j, t), "another tile's accumulator")
        yield ("arrive", f"empty{s}")

    for j in range(maps):
        for layer in range(3):
            for u in range(g, TILES, GROUPS):
                yield from read(j, layer * TILES + u)
                if layer == 1:
                    net.b[u] = ("layer2", j)
                else:
                    net.a[u] = (layer, j)
                yield ("arrive", f"stored{layer}_{u}")
            if layer == 0:
                yield ("meet",)
        for u in range(TILES):
            yield ("wait", f"stored2_{u}", j)
        for u in range(g, TILES, GROUPS):
            yield from read(j, 3 * TILES + u)
            net.b[u] = ("z", j)
        yield ("meet",)


def output(net, maps, made):
    def repack(j):
        need(net.stage == j, "another map's copy")
        net.first, net.stage = j, None

    def logits(j):
        # Reads z over some time, then B's groups are free.
        for u in range(TILES):
            need(net.b.get(u) == ("z", j), "the logits read z")
            yield ("go",)
        made.append(j)

    yield ("wait", "stage", 0)
    repack(0)
    yield ("arrive", "input")
    for j in range(maps):
        if j:
            yield from logits(j - 1)
        yield ("meet",)
        for u in range(TILES):
            yield ("wait", f"stored2_{u}", j)
        if j + 1 < maps:
            yield ("wait", "stage", j + 1)
            repack(j + 1)
            yield ("arrive", "input")
        yield ("meet",)
    yield from logits(maps - 1)


def run(maps, seed, issuers=ISSUERS, skip_meeting=None):
    rnd = random.Random(seed)
    net, made, phases = Net(), [], {}
    joined = [epilogue(net, g, maps) for g in range(GROUPS)] + [output(net, maps, made)]
    if skip_meeting is not None:
        joined = [drop(a, skip_meeting) for a in joined]
    agents = dict(enumerate(joined + [issuer(net, i, maps, issuers) for i in range(issuers)]))
    pace = {k: rnd.choice([1, 1, 5, 20]) for k in agents}
    cur = {k: next(a) for k, a in agents.items()}
    while agents:
        ready = []
        for k, op in cur.items():
            if op[0] in ("arrive", "go"):
                ready.append(k)
            elif op[0] == "wait":
                _, b, c = op
                n = phases.get(b, 0)
                if n > c + 1 or ((n & 1) != (c & 1)) != (n >= c + 1):
                    raise Wrong(f"parity: role {k} waits for phase {c} of {b}, {n} done")
                if n > c:
                    ready.append(k)
        if all(cur.get(k, ("gone",))[0] == "meet" for k in range(len(joined))):
            step = list(range(len(joined)))
        else:
            need(ready, f"deadlock: {cur}")
            step = [rnd.choices(ready, [pace[k] for k in ready])[0]]
        for k in step:
            if cur[k][0] == "arrive":
                phases[cur[k][1]] = phases.get(cur[k][1], 0) + 1
            try:
                cur[k] = next(agents[k])
            except StopIteration:
                del agents[k], cur[k]
    assert made == list(range(maps)) and not net.slots


def drop(agent, which):
    """The role without its first (0) or second (1) meeting of every map."""
    n = 0
    for op in agent:
        if op[0] == "meet":
            n += 1
            if (n - 1) % 2 == which:
                continue
        yield op


def test_constants_fit_the_roles():
    # A slot's tiles come from one issuer, and a barrier's arrivals are a group's warps.
    assert NSLOT % ISSUERS == 0 and GROUPS == 2 and GRP == 128
    kernel = TEXT[TEXT.index("lp_net_kernel("):TEXT.index("namespace lptrain")]
    assert kernel.count("ok = !out_or(!ok);") == 2  # the two meetings
    assert "tiles(j, 0, grp, 2);" in kernel and "for (int u = grp; grp < 2 && u < TILES && ok; u += 2)" in kernel


@pytest.mark.parametrize("maps", [1, 2, 4])
def test_roles_hand_over_in_order(maps):
    for seed in range(120):
        run(maps, seed)


@pytest.mark.parametrize("issuers", [1, 2, 8])
def test_roles_hold_for_other_issuer_counts(issuers):
    for seed in range(60):
        run(3, seed, issuers)


@pytest.mark.parametrize("which", [0, 1])
def test_the_check_catches_a_missing_meeting(which):
    with pytest.raises(Wrong):
        for seed in range(400):
            run(3, seed, skip_meeting=which)
