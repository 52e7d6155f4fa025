"""Simulation of the hand-offs in the core of the query-resident attention kernels (csrc/tkv_attn_pair.cuh) under random
interleavings, with the barriers and checks of ``test_linrec_protocol``.  Products complete in the order they were issued in only
where they have one accumulator, as PTX promises, and a commit arrives when everything its thread issued before is complete: a
score that overwrites weights which a product still reads, in whatever order the tensor core takes them, is a failure."""
import random

import pytest

from tests.test_linrec_protocol import Bar, Sim

LANES = (0, 1)          # two agents stand for the rows of a tile


class PairSim(Sim):
    def __init__(self, ranges, nk, nv, rng):
        super().__init__(max(r[1] for r in ranges), False, False, rng)
        self.ranges, self.nk, self.nv = ranges, nk, nv
        self.bar = {f"full_k{i}": Bar(1) for i in range(nk)} | {f"full_v{i}": Bar(1) for i in range(nv)}
        self.bar |= {f"empty_k{i}": Bar(1) for i in range(nk)} | {f"empty_v{i}": Bar(1) for i in range(nv)}
        self.bar |= {f"{k}{t}": Bar(1) for k in "so" for t in (0, 1)} | {f"{k}{t}": Bar(len(LANES)) for k in ("half", "ready") for t in (0, 1)}

    # ---- products and commits of the issuing thread: (resources read, accumulator, resources written, value) or a barrier
    def issue(self, reads, acc, writes, value):
        for r, chunk in reads:
            self.read(r, chunk)
            self.busy[r] = self.busy.get(r, 0) + 1
        for w in writes:
            self.write(w, ("writing", value))
        self.queues["main"].append(([r for r, _ in reads], acc, writes, value))

    def commit(self, bar):
        self.queues["main"].append(bar)
        if all(isinstance(e, str) for e in self.queues["main"]):
            self.queues["main"].pop()
            self.bar[bar].arrive()

    def complete(self, queue):
        if queue == "tma":
            return super().complete(queue)
        q = self.queues[queue]
        ops = [e for e in q if not isinstance(e, str)]
        reads, acc, writes, value = done = self.rng.choice([e for i, e in enumerate(ops) if all(e[1] != x[1] for x in ops[:i])])
        q.remove(done)
        for r in reads:
            self.busy[r] -= 1
        for w in writes:
            self.buf[w] = value
        while q and isinstance(q[0], str):
            self.bar[q.pop(0)].arrive()

    # ---- roles
    def copies(self):
        for i in range(self.n + 1):
            if i < self.n:
                yield from self.wait(f"empty_k{i % self.nk}", i // self.nk - 1)
                self.copy([f"K{i % self.nk}"], i, f"full_k{i % self.nk}")
                yield
            if i > 0:
                j = i - 1
                yield from self.wait(f"empty_v{j % self.nv}", j // self.nv - 1)
                self.copy([f"V{j % self.nv}"], j, f"full_v{j % self.nv}")
                yield

    def products(self):
        def lanes(part, t):
            return [f"{part}{t}.{a}" for a in LANES]
        for j in range(-1, self.n):
            jn = j + 1
            if j >= 0:
                yield from self.wait(f"full_v{j % self.nv}", j // self.nv)
            if jn < self.n:
                yield from self.wait(f"full_k{jn % self.nk}", jn // self.nk)
            give_v = j >= 0 and j + self.nv < self.n
            for t in (0, 1):
                j0, j1 = self.ranges[t]
                now, after = j0 <= j < j1, j0 <= jn < j1
                if now:
                    for half, bar in enumerate(("half", "ready")):
                        yield from self.wait(f"{bar}{t}", j - j0)
                        self.issue([(f"V{j % self.nv}", j)] + [(r, ("P", j)) for r in lanes(f"low{half}", t)], f"O{t}", [f"O{t}"], j)
                        yield
                    self.commit(f"o{t}")
                if self.nv == 1 and t == 1 and give_v:
                    self.commit(f"empty_v{j % self.nv}")
                yield
                if after:
                    if now:
                        yield from self.wait(f"o{t}", j - j0)
                    self.issue([(f"K{jn % self.nk}", jn)], f"S{t}", lanes("low0", t) + lanes("low1", t) + lanes("high", t), ("S", jn))
                    self.commit(f"s{t}")
                    yield
            if self.nv > 1 and give_v:
                self.commit(f"empty_v{j % self.nv}")
            if jn + self.nk < self.n:
                self.commit(f"empty_k{jn % self.nk}")
            yield

    def rows(self, t, a):
        j0, j1 = self.ranges[t]
        for j in range(j0, j1):
            yield from self.wait(f"s{t}", j - j0)
            for part in ("low0", "low1", "high"):
                self.read(f"{part}{t}.{a}", ("S", j))
                yield
            if j > j0:
                self.read(f"O{t}", j - 1)                           # rescaled by a thread of its own row: nothing may be adding to it
                assert not any(e[1] == f"O{t}" for e in self.queues["main"] if not isinstance(e, str))
            for half, bar in enumerate(("half", "ready")):
                yield
                self.write(f"low{half}{t}.{a}", ("P", j))
                yield
                self.bar[f"{bar}{t}"].arrive()
        if j1 > j0:
            yield from self.wait(f"o{t}", j1 - 1 - j0)
            self.read(f"O{t}", j1 - 1)

    def agents(self):
        return [self.copies(), self.products()] + [self.rows(t, a) for t in (0, 1) for a in LANES]

    def run(self):
        super().run()
        assert not any(self.queues.values())                        # nothing lands in the memory of a CTA that has gone


# key tiles of the two tiles of rows: a causal pair, both ends apart (a window), and one tile of rows that sees nothing
RANGES = [((0, 1), (0, 1)), ((0, 2), (0, 3)), ((0, 5), (0, 5)), ((0, 4), (1, 5)), ((2, 3), (0, 6)), ((0, 0), (0, 4)), ((0, 4), (0, 0))]


@pytest.mark.parametrize("stages", [(3, 2), (2, 2), (2, 1), (3, 1)])
@pytest.mark.parametrize("ranges", RANGES)
def test_hand_offs_hold_under_random_interleavings(ranges, stages):
    for seed in range(100):
        PairSim(ranges, *stages, random.Random(seed)).run()


# without the wait for P.V the scores of the next keys are written over weights that the product may still read
@pytest.mark.parametrize("missing", ["o", "half", "ready", "empty_v", "empty_k"])
def test_the_simulation_notices_a_missing_wait(missing):
    class Broken(PairSim):
        def wait(self, name, phase):
            if name.startswith(missing) and not (missing == "o" and phase == 4):      # the epilogue's wait stays
                return
            yield from super().wait(name, phase)
    with pytest.raises(AssertionError):
        for seed in range(300):
            Broken(((0, 5), (0, 5)), 2, 1, random.Random(seed)).run()
