"""The lean prepare kernel's roles as a model on the CPU (gdn_chunk_prepare_lean_sm100.cu): mbarriers with their counts and parities, copies and products that end whenever
they like, and every role's waits and arrivals in the order of the code, under a random scheduler that makes some roles slow.  A run fails when no role can go on, when a wait
by parity lets a role through a phase early, or when a buffer is written or read out of order.  (A cycle of waits
through SQ and LOW and a missing order were found so.)"""

import random

import pytest


class Barrier:
    def __init__(self, count):
        self.count, self.arrived, self.pending, self.phase = count, 0, 0, 0

    def update(self, arrived=0, pending=0):
        self.arrived += arrived
        self.pending += pending
        if self.arrived == self.count and self.pending == 0:
            self.arrived = 0
            self.phase += 1


class Model:
    """heads: value heads per CTA; items: of this CTA.  Roles are generators: they yield None (anything may happen in between) or (barrier, item) to wait for."""

    def __init__(self, heads, l2norm, items):
        self.H, self.l2, self.n = heads, l2norm, items
        counts = {"K": 1, "Q": 1, "MMA": 1, "ENT": 4 * heads, "SQ": 3 * heads}
        for h in range(heads):
            counts.update({("TAB", h): 2 if l2norm else 1, ("PAIR", h): 2, ("EXF", h): 2, ("EXE", h): 2, ("LOW", h): 1})
        self.bars = {name: Barrier(c) for name, c in counts.items()}
        self.done = {("item", h, i) for h in range(heads) for i in (0, 1)}
        self.flight = []                     # copies and products under way

    def need(self, *events):
        for e in events:
            assert e in self.done, ("not yet", e)

    def never(self, *events):
        for e in events:
            assert e not in self.done, ("too late for", e)

    def arrive(self, bar):
        self.bars[bar].update(arrived=1)

    def enter(self, h, i):
        yield (("TAB", h), i)
        yield ("MMA", i)
        self.arrive("ENT")

    def squares(self, h, role, i):
        yield ("KQ"[role], i)
        self.need(("loaded", "KQ"[role], i))
        self.never(("loaded", "K", i + 2), ("loaded", "Q", i + 2))
        yield None
        self.done.add(("squares", h, role, i))
        self.arrive("SQ")

    def norms(self, h, i):
        yield ("SQ", i)
        self.need(("gates", h, i), *[("squares", x, r, i) for x in range(self.H) for r in (0, 1)])
        yield None
        self.arrive(("TAB", h))

    def diagonal(self, h, role):             # roles 0 and 1
        if self.l2:
            yield from self.squares(h, role, 0)
        for i in range(self.n):
            yield from self.enter(h, i)
            self.need(("gates", h, i))
            if i > 1:
                self.need(("scalars", h, i - 2))           # the bound of two items before has been read
            yield None
            self.done.add(("mask", h, role, i))
            if self.l2 and i + 1 < self.n:
                yield from self.squares(h, role, i + 1)
            if i > 0:
                yield (("EXE", h), i - 1)
                self.need(("below", h, 2, i - 1), ("below", h, 3, i - 1))
            yield None
            self.done.add(("published", h, role, i))
            self.arrive(("EXF", h))
            yield None
            self.done.add(("diagonal", h, role, i))

    def below(self, h, role, i):
        yield (("EXF", h), i)
        self.need(("published", h, 0, i), ("published", h, 1, i))
        self.never(("published", h, 0, i + 1), ("published", h, 1, i + 1))
        if role == 2:
            self.done.add(("scalars", h, i))
        elif i > 0:
            self.need(("stored", h, i - 1), ("left", h, i - 1))
        yield None
        self.done.add(("below", h, role, i))
        self.arrive(("EXE", h))

    def role2(self, h):
        for i in range(self.n + 2):
            more, one = i < self.n, 0 < i <= self.n
            if one:
                yield from self.enter(h, i - 1)
            if more and h == 0:
                self.need(("item", 0, i), *([("product", i - 1)] if i else []))
                if i and self.l2:
                    self.need(*[("squares", x, 0, i - 1) for x in range(self.H)])
                self.flight.append(("K", i))
                self.bars["K"].update(pending=1)
                self.bars["Q"].update(pending=self.H)
                self.arrive("K")
                self.arrive("Q")
            yield None
            if one:
                self.done.add(("P", h, 2, i - 1))
                yield None
                if i + 1 < self.n:
                    if i >= 3:
                        self.need(("below", h, 3, i - 3), ("stored", h, i - 3))
                    self.done.add(("item", h, i + 1))
            if i > 0:
                self.done.add(("left", h, i - 3))          # its own copies out have been read
                self.arrive(("PAIR", h))
                yield (("PAIR", h), i - 1)
                if one:
                    self.need(("P", h, 3, i - 1))
            if more:
                if i:
                    self.need(("product", i - 1))
                    if self.l2:
                        self.need(*[("squares", x, 1, i - 1) for x in range(self.H)])
                self.flight.append(("Q", i))
            yield None
            if i > 1:
                yield from self.below(h, 2, i - 2)
                yield (("LOW", h), i - 2)
                self.need(("below", h, 3, i - 2))
                self.done.add(("stored", h, i - 2))
            if more:
                if h == 0:
                    if one:
                        yield ("ENT", i - 1)
                    yield ("K", i)
                    yield ("Q", i)
                    if i > 1:                              # the accumulator of two items before
                        self.need(*[(e, x, r, i - 2) for x in range(self.H) for e, r in (("mask", 0), ("mask", 1), ("P", 2), ("P", 3))])
                    self.need(("loaded", "K", i), ("loaded", "Q", i))
                    self.flight.append(("MMA", i))
                if self.l2:
                    yield from self.norms(h, i)

    def role3(self, h):
        for i in range(self.n + 2):
            more, one = i < self.n, 0 < i <= self.n
            if one:
                yield from self.enter(h, i - 1)
            if more:
                self.need(("item", h, i))
            if one:
                yield None
                self.done.add(("P", h, 3, i - 1))
            if i > 0:
                self.arrive(("PAIR", h))
            if more:
                if one:
                    yield ("ENT", i - 1)
                    if i > 1:                              # tables of two items before, beta of four
                        self.need(("diagonal", h, 0, i - 2), ("diagonal", h, 1, i - 2), ("P", h, 2, i - 2))
                    if i > 3:
                        self.need(("below", h, 2, i - 4), ("below", h, 3, i - 4))
                yield None
                self.done.add(("gates", h, i))
                self.arrive("SQ" if self.l2 else ("TAB", h))
            if i > 0:
                yield (("PAIR", h), i - 1)
            if i > 1:
                yield from self.below(h, 3, i - 2)
                yield None
                self.arrive(("LOW", h))
            if more and self.l2:
                yield from self.norms(h, i)

    def end(self, kind, i):                                # of a copy or product
        if kind == "MMA":
            self.done.add(("product", i))
            self.arrive("MMA")
        else:
            left = self.bars[kind].pending
            if kind == "K" or left == 1:
                self.done.add(("loaded", kind, i))
            self.bars[kind].update(pending=-1)

    def run(self, rng):
        roles = [r for h in range(self.H) for r in (self.diagonal(h, 0), self.diagonal(h, 1), self.role2(h), self.role3(h))]
        weight = [1 / rng.choice([1, 1, 1, 20]) for _ in roles]
        at = {}

        def step(k):
            try:
                at[k] = next(roles[k])
            except StopIteration:
                at.pop(k, None)

        for k in range(len(roles)):
            step(k)
        while at:
            ready = [k for k, w in at.items() if w is None or (self.bars[w[0]].phase & 1) != (w[1] & 1)]
            events = ready + list(self.flight)
            assert events, ("no role can go on", dict(at))
            what = rng.choices(events, [weight[k] for k in ready] + [0.5] * len(self.flight))[0]
            if isinstance(what, tuple):
                self.flight.remove(what)
                self.end(*what)
            else:
                if at[what] is not None:
                    bar, item = at[what]
                    assert self.bars[bar].phase == item + 1, ("through a wait early or too late", bar, item, self.bars[bar].phase)
                step(what)
        assert all(b.arrived == 0 and b.pending == 0 for b in self.bars.values())


@pytest.mark.parametrize("heads", [1, 2])
@pytest.mark.parametrize("l2norm", [False, True])
def test_roles_of_the_prepare_kernel(heads, l2norm):
    for seed in range(400):
        rng = random.Random(seed)
        Model(heads, l2norm, rng.randint(1, 9)).run(rng)


@pytest.mark.parametrize("heads", [1, 2])
def test_the_model_finds_a_missing_order(heads):
    """Without the wait for all readers of an accumulator, or for the exchange's, some run fails."""
    class NoEnt(Model):
        def role2(self, h):
            return (w for w in super(NoEnt, self).role2(h) if w is None or w[0] != "ENT")

    class NoExe(Model):
        def diagonal(self, h, role):
            return (w for w in super(NoExe, self).diagonal(h, role) if w is None or w[0] != ("EXE", h))

    for kind in (NoEnt, NoExe):
        failed = 0
        for seed in range(200):
            rng = random.Random(seed)
            try:
                kind(heads, False, 6).run(rng)
            except AssertionError:
                failed += 1
        assert failed
