"""The rings of the converted-e4m3 pipeline as a CPU model: a lead that hands out
items and waits for every group's slot, four B issuers that copy groups ahead and
convert them, two MMA threads and four epilogue warps, on barriers with the
parity test of an mbarrier. The rules that the roles share are the kernel's own
(csrc/ring_rules.h, compiled here). Every schedule has to end: random ones, and
ones in which one role is starved whenever another can run. No GPU needed."""
import ctypes
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matrixmultiplicationcuda_gb300", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src = d / "rules.cpp"
    src.write_text('#include "ring_rules.h"\nextern "C" {\nint entries() { return spmm::kItemRing; }\n'
                   'int issuers() { return spmm::kBIssuers; }\n'
                   'int arrivals() { return spmm::kConvertFullArrivals; }\n'
                   'int may_wait(unsigned converted, unsigned first) { return spmm::may_wait_for_entry(converted, first); }\n}\n')
    so = d / "rules.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


class Barrier:
    def __init__(self, arrivals):
        self.arrivals = self.left = arrivals
        self.phase = 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left = self.arrivals
            self.phase += 1

    def passed(self, parity):
        return (self.phase & 1) != parity


class Deadlock(Exception):
    pass


class Cta:
    """items: groups of each item of one CTA, in order. A role yields the barrier
    and parity that it waits for."""

    def __init__(self, rules, items, stages, arrivals=None, may_wait=None):
        self.items, self.stages = items, stages
        self.may_wait = may_wait or rules.may_wait
        self.Q, self.issuers = rules.entries(), rules.issuers()
        arrivals = rules.arrivals() if arrivals is None else arrivals
        self.lead_arrives = arrivals > self.issuers
        self.full = [Barrier(arrivals) for _ in range(stages)]
        self.empty = [Barrier(2) for _ in range(stages)]
        self.tfull, self.tempty = [Barrier(2) for _ in range(2)], [Barrier(4) for _ in range(2)]
        self.qfull = [Barrier(1) for _ in range(self.Q)]
        self.qempty = [Barrier(2 + self.issuers + 4) for _ in range(self.Q)]
        self.ring = [None] * self.Q
        self.slot = [[-1] * self.issuers for _ in range(stages)]   # group that each issuer has put there
        self.used = [0, 0]                                         # groups that each MMA thread has read

    def publish(self, e, groups):
        if e >= self.Q:
            yield self.qempty[e % self.Q], (e // self.Q + 1) & 1
        self.ring[e % self.Q] = groups
        self.qfull[e % self.Q].arrive()

    def read(self, e):
        yield self.qfull[e % self.Q], (e // self.Q) & 1
        groups = self.ring[e % self.Q]
        self.qempty[e % self.Q].arrive()
        return groups

    def lead(self):
        items = self.items + [-1]
        gs, published = 0, False
        for it, groups in enumerate(items):
            if not published:
                yield from self.publish(it, groups)
            if groups < 0:
                return
            claimed = published = False
            for gi in range(groups):
                if not published:
                    if claimed:
                        yield from self.publish(it + 1, items[it + 1])
                        published = True
                    elif groups - gi <= self.stages:
                        claimed = True
                s = gs % self.stages
                if gs >= self.stages:
                    yield self.empty[s], (gs // self.stages + 1) & 1
                if self.lead_arrives:
                    self.full[s].arrive()
                gs += 1

    def issuer(self, me):
        it = left = copied = gs = 0
        done, first = False, [0] * self.Q   # first group of each entry of the item ring
        while True:
            while copied - gs < self.stages:
                while not done and left == 0 and self.may_wait(gs, first[it % self.Q]):
                    first[it % self.Q] = copied
                    left = yield from self.read(it)
                    it += 1
                    done = left < 0
                if done or left == 0:
                    break
                left -= 1
                copied += 1
            if copied == gs:
                assert done
                return
            s = gs % self.stages
            if gs >= self.stages:
                yield self.empty[s], (gs // self.stages + 1) & 1
            assert min(self.used) > gs - self.stages, "a slot overwritten before it was read"
            self.slot[s][me] = gs
            self.full[s].arrive()
            gs += 1

    def mma(self, me):
        gs = it = 0
        while True:
            groups = yield from self.read(it)
            if groups < 0:
                return
            if it >= 2:
                yield self.tempty[it % 2], (it // 2 + 1) & 1
            for _ in range(groups):
                s = gs % self.stages
                yield self.full[s], (gs // self.stages) & 1
                assert self.slot[s] == [gs] * self.issuers, "a slot read before it was filled"
                gs += 1
                self.used[me] = gs
                self.empty[s].arrive()
            self.tfull[it % 2].arrive()
            it += 1

    def epilogue(self):
        it = 0
        while (yield from self.read(it)) >= 0:
            yield self.tfull[it % 2], (it // 2) & 1
            self.tempty[it % 2].arrive()
            it += 1

    def run(self, rng, starved):
        """starved: index of a role that runs only when no other can (-1: none)."""
        roles = [self.lead()] + [self.issuer(i) for i in range(self.issuers)] + [self.mma(0), self.mma(1)]
        roles += [self.epilogue() for _ in range(4)]
        waits = {}
        for r in roles:
            waits[r] = next(r, None)
        live = [r for r in roles if waits[r] is not None]
        while live:
            ready = [r for r in live if waits[r][0].passed(waits[r][1])]
            if not ready:
                raise Deadlock()
            others = [r for r in ready if starved < 0 or r is not roles[starved]]
            r = rng.choice(others or ready)
            waits[r] = next(r, None)
            if waits[r] is None:
                live.remove(r)


def run_all(rules, items, stages, **kw):
    for starved in range(-1, 11):
        for seed in range(2):
            Cta(rules, items, stages, **kw).run(random.Random(seed), starved)


# groups in flight: two (32-row blocks) or three (64-row blocks)
@pytest.mark.parametrize("stages", [2, 3])
@pytest.mark.parametrize("items", [[1], [9], [1] * 12, [20, 1, 20, 1], [7, 2, 3, 1, 4, 11, 5], [13] * 5])
def test_items_with_blocks(rules, items, stages):
    run_all(rules, items, stages)


@pytest.mark.parametrize("stages", [2, 3])
def test_a_lead_that_waits_without_arriving_is_left_behind(rules, stages):
    with pytest.raises(Deadlock):
        run_all(rules, [20, 1], stages, arrivals=rules.issuers())


# items without blocks: after a long row, at the end, between rows of one group, everywhere
@pytest.mark.parametrize("stages", [2, 3])
@pytest.mark.parametrize("items", [[5, 0, 0, 0, 0], [1] + [0] * 16 + [1], [0] * 9, [20] + [0] * 5 + [3] + [0] * 4 + [1, 2],
                                   [3, 0, 1, 0, 0, 1, 0, 0, 4], [1, 0, 1, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 0, 1]])
def test_items_without_blocks(rules, items, stages):
    run_all(rules, items, stages)


def test_random_items(rules):
    for seed in range(400):
        rng = random.Random(seed)
        items = [rng.choice((0, 0, 0, 1, 1, 2, 3, 5)) for _ in range(rng.randrange(1, 24))]
        Cta(rules, items, rng.choice((2, 3))).run(rng, rng.randrange(-1, 11))


@pytest.mark.parametrize("stages,items", [(2, [1, 0, 0, 0, 0]), (3, [1, 0, 0, 0, 0]), (3, [3, 0, 1, 0, 0, 1, 0, 0, 4])])
def test_an_issuer_that_always_waits_for_the_next_item_waits_for_itself(rules, stages, items):
    with pytest.raises(Deadlock):
        run_all(rules, items, stages, may_wait=lambda converted, first: True)
