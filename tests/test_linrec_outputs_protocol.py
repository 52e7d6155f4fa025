"""The hand-offs of the tcgen05 recurrence kernel (csrc/tkv_linrec_tc.cu) as they are now: two stages of Q and K, weights over the scores
in TMEM, a chunk's outputs behind the next chunk's weighted values; a whole chunk's outputs take the place of its values and are
copied out of there.  Barriers, checks and asynchronous products are those of
``test_linrec_protocol``, whose roles are an earlier order of the same work."""
import random

import pytest

from tests.test_linrec_protocol import Bar, Sim


class LaterOutputs(Sim):
    def __init__(self, nchunks, state_only, partial, rng):
        super().__init__(nchunks, state_only, partial, rng)
        self.bar["out"], self.bar["stored"] = Bar(2), Bar(1)
        self.queues["store"] = []
        self.bar |= {"qk0": Bar(1), "qk1": Bar(1)}

    def issue(self, reads, outs, chunk, bar):
        """A product of operands ``(resource, what it holds)``."""
        for r, holds in reads:
            self.read(r, holds)
            self.busy[r] = self.busy.get(r, 0) + 1
        for o in outs[:-1]:
            self.write(o, ("writing", chunk))
            self.queues["main"].append(([], o, chunk, None))
        self.write(outs[-1], ("writing", chunk))
        self.queues["main"].append(([r for r, _ in reads], outs[-1], chunk, bar))

    def load_qk(self, i):
        self.copy([f"K{i & 1}"] if self.so else [f"Q{i & 1}", f"K{i & 1}"], i, f"qk{i & 1}")

    def store(self, i):
        for a in (0, 1):
            self.read(f"out{i & 1}{a}", i)
        self.product("store", [f"V{i & 1}"], f"tokens{i}", i, "stored")

    def control(self):
        self.load_qk(0)
        self.load_v(0)
        for i in range(self.n):
            q, k = (f"Q{i & 1}", i), (f"K{i & 1}", i)
            yield from self.wait(f"qk{i & 1}", i >> 1)
            if not self.so and i > 0:
                yield from self.wait("o2", i - 1)
            if i == self.n - 1 and self.partial:
                yield from self.wait("clr", 0)
            if not self.so:
                self.issue([q, k], ["S0", "S1"], i, "s")
                yield
            if i + 1 < self.n:
                if i > 0:
                    yield from self.wait("st", i - 1)
                    if not self.so:
                        yield from self.wait("o1", i - 1)
                self.load_qk(i + 1)
                yield
            yield from self.wait("sp", i)
            if self.so and i + 1 < self.n:
                self.load_v(i + 1)
                yield
            yield from self.wait("wv", i)
            self.issue([k, ("WV", i)], ["ST"], i, "st")
            yield
            if not self.so:
                if i > 0:
                    yield from self.wait("out", i - 1)
                self.issue([q, ("SP", i)], ["O1"], i, "o1")
                if i > 0:
                    self.store(i - 1)
                    yield
                    yield from self.wait("stored", i - 1)
                if i + 1 < self.n:
                    self.load_v(i + 1)
                yield
                yield from self.wait("p", i)
                self.issue([("S0", ("P", i)), ("S1", ("P", i)), (f"V{i & 1}", i)], ["O2"], i, "o2")
                yield
        if not self.so and not self.partial:
            yield from self.wait("out", self.n - 1)
            self.store(self.n - 1)

    def outputs(self, i, a):
        yield from self.wait("o2", i)
        for res in ("O1", "O2", f"V{i & 1}"):              # the row's decay is in a register
            self.read(res, i)
            yield
        if i < self.n - 1 or not self.partial:
            assert not self.busy.get(f"V{i & 1}"), f"outputs of chunk {i} over values that a product reads"
            self.write(f"out{i & 1}{a}", i)
            yield
        self.bar["out"].arrive()
        yield

    def half(self, a):
        for i in range(self.n):
            if i == self.n - 1 and self.partial:
                yield from self.wait(f"qk{i & 1}", i >> 1)
                yield from self.wait(f"v{i & 1}", i >> 1)
                self.write(f"K{i & 1}", i)
                self.write(f"V{i & 1}", i)
                yield
                self.bar["clr"].arrive()
                yield
            yield from self.wait(f"l{i & 1}", i >> 1)
            if i > 0:
                yield from self.wait("st", i - 1)
                if not self.so:
                    yield from self.wait("o1", i - 1)
                self.read("ST", i - 1)
            self.read(f"L{i & 1}", i)
            if not self.so:
                self.write("SP", i)
                yield
            self.bar["sp"].arrive()
            yield
            yield from self.wait(f"v{i & 1}", i >> 1)
            self.read(f"V{i & 1}", i)
            self.read(f"L{i & 1}", i)
            self.write("WV", i)
            yield
            self.bar["wv"].arrive()
            yield
            if self.so:
                continue
            if i > 0:
                yield from self.outputs(i - 1, a)
            yield from self.wait("s", i)
            self.read(f"S{a}", i)
            yield
            self.read(f"L{i & 1}", i)
            self.write(f"S{a}", ("P", i))
            yield
            self.bar["p"].arrive()
            yield
        if not self.so:
            yield from self.wait("o1", self.n - 1)
            yield from self.outputs(self.n - 1, a)
        yield from self.wait("st", self.n - 1)
        self.read("ST", self.n - 1)

    def agents(self):
        return [self.control(), self.scan(), self.half(0), self.half(1)]


@pytest.mark.parametrize("state_only", [False, True])
@pytest.mark.parametrize("nchunks", [1, 2, 3, 4, 9])
def test_hand_offs_hold_under_random_interleavings(nchunks, state_only):
    for seed in range(200):
        rng = random.Random(1000 * nchunks + seed)
        LaterOutputs(nchunks, state_only, partial=not state_only and bool(seed & 1), rng=rng).run()


@pytest.mark.parametrize("missing", ["out", "o1", "o2", "p", "stored"])
def test_the_simulation_notices_a_missing_wait(missing):
    class Broken(LaterOutputs):
        def wait(self, name, phase):
            if name == missing:
                return
            yield from super().wait(name, phase)
    with pytest.raises(AssertionError):
        for seed in range(300):
            Broken(6, False, False, random.Random(seed)).run()
