"""Model check of the mbarrier protocols of the tcgen05 attention kernels (csrc/attn_bwd_tcgen05.cu, attn_fwd_bias.cu; with the simulator for
csrc/attn_fwd_tcgen05.cu, whose roles are in test_attention_forward_protocol_cpu.py).

The roles of a CTA (TMA producer and scheduler, MMA issuer, softmax / element warps) are written as coroutines that perform exactly the waits,
arrives, expect_tx and commits of the kernels (same barrier names, same parities), over several work items of one CTA where the kernel is
persistent; TMA completions, answers to requests for further items and tensor-pipe completions are asynchronous events.  A randomised scheduler
interleaves everything over many seeds and checks
  * no deadlock (every role finishes) and no parity aliasing (a wait never needs a phase that is two completions away),
  * no buffer hazard: a shared-memory stage / TMEM buffer / item slot is never overwritten before its consumers released it and never
    read before it was produced.  Buffers without a barrier of their own (P over S, which the next products overwrite) rely on the
    tensor pipe's order, which the model keeps.
This is the part of the kernels that cannot be unit-tested without hardware and whose failure mode on hardware is a hang."""
import random

import pytest


class Bar:
    def __init__(self, count):
        self.init, self.count, self.tx, self.phase = count, count, 0, 0

    def _check(self):
        if self.count == 0 and self.tx == 0:
            self.phase += 1
            self.count = self.init

    def arrive(self):
        assert self.count > 0, "more arrivals than the barrier expects in one phase"
        self.count -= 1
        self._check()

    def expect_tx(self, n):      # mbarrier.arrive.expect_tx
        self.tx += n
        self.arrive()

    def complete_tx(self, n):
        self.tx -= n
        assert self.tx >= 0
        self._check()

    def passed(self, parity):   # mbarrier.try_wait.parity
        return (self.phase & 1) != parity


class Sim:
    """Roles are generators yielding ("wait", bar_name, parity); everything else they do is immediate."""

    def __init__(self, seed, bars):
        self.rng = random.Random(seed)
        self.bars = {k: Bar(c) for k, c in bars.items()}
        self.pipe = []      # tensor pipe: in-order list of callables (MMA effects, commits)
        self.tma = []       # outstanding TMA loads: callables, complete in any order
        self.state = {}     # buffer name -> "free" | "loading" | "full"

    # ---- buffer hazard tracking
    def expect(self, buf, want, what):
        got = self.state.get(buf, "free")
        assert got == want, f"{what}: buffer {buf} is {got}, expected {want}"

    def set(self, buf, st):
        self.state[buf] = st

    def run(self, roles):
        blocked = {name: None for name in roles}
        gens = dict(roles)
        steps = 0
        while gens or self.pipe or self.tma:
            steps += 1
            assert steps < 200000, "livelock"
            choices = []
            for name, g in gens.items():
                w = blocked[name]
                if w is None or self.bars[w[0]].passed(w[1]):
                    choices.append(("role", name))
            if self.pipe:
                choices.append(("pipe", None))
            for i in range(len(self.tma)):
                choices.append(("tma", i))
            if not choices:
                waiting = {n: blocked[n] for n in gens}
                raise AssertionError(f"deadlock: {waiting}, phases { {k: b.phase for k, b in self.bars.items()} }")
            kind, arg = self.rng.choice(choices)
            if kind == "pipe":
                self.pipe.pop(0)()
            elif kind == "tma":
                self.tma.pop(arg)()
            else:
                blocked[arg] = None
                try:
                    req = next(gens[arg])
                    assert req[0] == "wait"
                    blocked[arg] = (req[1], req[2])
                except StopIteration:
                    del gens[arg]


# ------------------------------------------------------------------------------------------------ forward kernel with a learned bias
def fwd_protocol(sim: Sim, n_kv: int):
    B = sim.bars
    KV = 100  # bytes of one K or V stage (any positive number)

    def producer():
        B["Q_FULL"].expect_tx(50)
        sim.expect("Q", "free", "Q load"); sim.set("Q", "loading")
        sim.tma.append(lambda: (sim.set("Q", "full"), B["Q_FULL"].complete_tx(50)))
        for j in range(n_kv):
            st, par = j & 1, (j >> 1) & 1
            for nm in ("K", "V"):
                yield ("wait", f"{nm}_EMPTY{st}", par ^ 1)
                B[f"{nm}_FULL{st}"].expect_tx(KV)
                sim.expect(f"{nm}{st}", "free", f"{nm} load of tile {j}"); sim.set(f"{nm}{st}", "loading")
                sim.tma.append(lambda nm=nm, st=st: (sim.set(f"{nm}{st}", "full"), B[f"{nm}_FULL{st}"].complete_tx(KV)))

    def mma():
        def issue_s(j):
            st, par = j & 1, (j >> 1) & 1
            yield ("wait", f"K_FULL{st}", par)
            yield ("wait", f"S_EMPTY{st}", par ^ 1)

            def exec_s():
                sim.expect("Q", "full", "S mma"); sim.expect(f"K{st}", "full", f"S mma {j}")
                sim.expect(f"S{st}", "free", f"S mma {j} overwrites S buffer"); sim.set(f"S{st}", "full")
            sim.pipe.append(exec_s)
            sim.pipe.append(lambda: (sim.set(f"K{st}", "free"), B[f"K_EMPTY{st}"].arrive()))
            sim.pipe.append(lambda: B[f"S_FULL{st}"].arrive())
        yield ("wait", "Q_FULL", 0)
        yield from issue_s(0)
        for j in range(n_kv):
            if j + 1 < n_kv:
                yield from issue_s(j + 1)
            st, par = j & 1, (j >> 1) & 1
            yield ("wait", "P_FULL", j & 1)
            yield ("wait", f"V_FULL{st}", par)
            yield ("wait", f"O_EMPTY{st}", par ^ 1)

            def exec_pv(st=st, j=j):
                sim.expect("P", "full", f"PV mma {j}"); sim.expect(f"V{st}", "full", f"PV mma {j}")
                sim.expect(f"T{st}", "free", f"PV mma {j} overwrites T buffer"); sim.set(f"T{st}", "full")
            sim.pipe.append(exec_pv)
            sim.pipe.append(lambda st=st: (sim.set(f"V{st}", "free"), B[f"V_EMPTY{st}"].arrive()))
            sim.pipe.append(lambda: (sim.set("P", "free"), B["P_EMPTY"].arrive()))
            sim.pipe.append(lambda st=st: B[f"O_FULL{st}"].arrive())

    def softmax(w):
        def fold(t):
            b = t & 1
            yield ("wait", f"O_FULL{b}", (t >> 1) & 1)
            sim.expect(f"T{b}", "full", f"fold {t}")
            sim.state[f"T{b}_readers"] = sim.state.get(f"T{b}_readers", 0) + 1
            if sim.state[f"T{b}_readers"] == 4:   # the buffer is free once all four warps arrived
                sim.state[f"T{b}_readers"] = 0
                sim.set(f"T{b}", "free")
            B[f"O_EMPTY{b}"].arrive()
        for j in range(n_kv):
            b = j & 1
            yield ("wait", f"S_FULL{b}", (j >> 1) & 1)
            sim.expect(f"S{b}", "full", f"softmax {j} pass 1")
            if j > 0:
                yield ("wait", "P_EMPTY", (j - 1) & 1)
            sim.expect(f"S{b}", "full", f"softmax {j} pass 2")
            sim.expect("P", "free" if w == 0 or sim.state.get("P_writers", 0) == 0 else "free", f"P write {j}")
            sim.state["P_writers"] = sim.state.get("P_writers", 0) + 1
            sim.state[f"S{b}_readers"] = sim.state.get(f"S{b}_readers", 0) + 1
            if sim.state[f"S{b}_readers"] == 4:
                sim.state[f"S{b}_readers"] = 0
                sim.set(f"S{b}", "free")
            if sim.state["P_writers"] == 4:
                sim.state["P_writers"] = 0
                sim.set("P", "full")
            B[f"S_EMPTY{b}"].arrive()
            B["P_FULL"].arrive()
            if j > 0:
                yield from fold(j - 1)
        yield from fold(n_kv - 1)

    roles = {"producer": producer(), "mma": mma()}
    for w in range(4):
        roles[f"softmax{w}"] = softmax(w)
    return roles


FWD_BARS = {"Q_FULL": 1, "P_FULL": 4, "P_EMPTY": 1}
for _st in (0, 1):
    FWD_BARS.update({f"K_FULL{_st}": 1, f"K_EMPTY{_st}": 1, f"V_FULL{_st}": 1, f"V_EMPTY{_st}": 1, f"S_FULL{_st}": 1,
                     f"S_EMPTY{_st}": 4, f"O_FULL{_st}": 1, f"O_EMPTY{_st}": 4})


@pytest.mark.parametrize("n_kv", [1, 2, 3, 4, 5, 8])
def test_forward_protocol_has_no_deadlock_or_buffer_hazard(n_kv):
    for seed in range(150):
        sim = Sim(seed, FWD_BARS)
        sim.run(fwd_protocol(sim, n_kv))
        assert all(v in ("free", "full", 0) for v in sim.state.values())


# ------------------------------------------------------------------------------------------------ persistent kernels: items
def count_down(sim, key, n):
    """True for the last of n callers."""
    sim.state[key] = sim.state.get(key, 0) + 1
    if sim.state[key] == n:
        sim.state[key] = 0
        return True
    return False


class Items:
    """The two item slots between the scheduler and its readers, and the requests for further items (one outstanding at a time)."""

    def __init__(self, sim, items, readers):
        self.sim, self.items, self.readers, self.n_pub, self.n_req = sim, items, readers, 0, 0
        self.slots, self.answer, self.asked = [None, None], None, 0

    def request(self):
        assert self.answer is None, "an answer is overwritten before it was read"
        self.sim.bars["CLC_FULL"].expect_tx(16)
        self.asked += 1

        def land(i=self.asked):
            self.answer = (i,)
            self.sim.bars["CLC_FULL"].complete_tx(16)
        self.sim.tma.append(land)

    def next(self):                                  # -> the next item's number, or None
        yield ("wait", "CLC_FULL", self.n_req & 1)
        self.n_req += 1
        (i,), self.answer = self.answer, None
        return i if i < len(self.items) else None

    def publish(self, item):
        slot = self.n_pub & 1
        yield ("wait", f"IT_EMPTY{slot}", ((self.n_pub >> 1) & 1) ^ 1)
        self.sim.expect(f"item{slot}", "free", f"item {self.n_pub} published")
        self.sim.set(f"item{slot}", "full")
        self.slots[slot] = (self.n_pub, item)
        self.sim.bars[f"IT_FULL{slot}"].arrive()
        self.n_pub += 1

    def take(self, n_it):
        slot = n_it & 1
        yield ("wait", f"IT_FULL{slot}", (n_it >> 1) & 1)
        n, item = self.slots[slot]
        assert n == n_it, f"slot {slot} holds item {n}, read as item {n_it}"
        if count_down(self.sim, f"item{slot}_readers", self.readers):
            self.sim.set(f"item{slot}", "free")
        self.sim.bars[f"IT_EMPTY{slot}"].arrive()
        return item


def load(sim, buf, bar, parts, what):
    sim.bars[bar].expect_tx(10 * parts)
    sim.expect(buf, "free", what)
    sim.set(buf, "loading")
    done = []

    def part():                                      # the boxes of a tile complete independently
        done.append(1)
        if len(done) == parts:
            sim.set(buf, "full")
        sim.bars[bar].complete_tx(10)
    for _ in range(parts):
        sim.tma.append(part)


ITEM_BARS = {"IT_FULL0": 1, "IT_FULL1": 1, "IT_EMPTY0": 9, "IT_EMPTY1": 9, "CLC_FULL": 1}


# The forward kernel's walk (its roles: test_attention_forward_protocol_cpu.py): stages of its K / V ring, which of a pair's query tiles takes a key tile
STAGES = 4
ONE, BOTH, SECOND = (True, False), (True, True), (False, True)


# ------------------------------------------------------------------------------------------------ backward kernel (both passes)
X_STAGES = 3


def bwd_protocol(sim: Sim, items, r_empty_parity=lambda n_pub: n_pub & 1):
    """An item is its number of steps."""
    B = sim.bars
    it = Items(sim, items, 9)

    def producer():
        g, idx = 0, 0
        it.request()
        while idx is not None:
            yield from it.publish(items[idx])
            yield ("wait", "R_EMPTY", r_empty_parity(it.n_pub))
            load(sim, "R", "R_FULL", 4, "resident tiles")
            for _ in range(items[idx]):
                st = g % X_STAGES
                yield ("wait", f"X_EMPTY{st}", ((g // X_STAGES) & 1) ^ 1)
                load(sim, f"X{st}", f"X_FULL{st}", 4, f"streamed tile {g}")
                g += 1
            idx = yield from it.next()
            if idx is not None:
                it.request()
        yield from it.publish(None)

    def mma():
        def issue_sdp(g, last):
            st, b = g % X_STAGES, g & 1
            yield ("wait", f"X_FULL{st}", (g // X_STAGES) & 1)

            def run():
                sim.expect("R", "full", "S / dP mma"), sim.expect(f"X{st}", "full", "S / dP mma"), sim.expect(f"S{b}", "free", "S / dP mma")
                sim.set(f"S{b}", "s")
            sim.pipe.append(run)
            sim.pipe.append(lambda: B[f"S_FULL{b}"].arrive())
            if last:
                sim.pipe.append(lambda: (sim.set("R", "free"), B["R_EMPTY"].arrive()))
        g, n_it = 0, 0
        while True:
            n = yield from it.take(n_it)
            if n is None:
                return
            yield ("wait", "R_FULL", n_it & 1)
            yield from issue_sdp(g, n == 1)
            for t in range(n):
                if t + 1 < n:
                    yield from issue_sdp(g + 1, t + 2 == n)
                st, b = g % X_STAGES, g & 1
                yield ("wait", f"P_FULL{b}", (g >> 1) & 1)
                if t == 0:
                    yield ("wait", "ACC_EMPTY", (n_it & 1) ^ 1)

                def run(st=st, b=b, was="acc" if t else "free"):
                    sim.expect(f"S{b}", "p", "accumulating mma"), sim.expect(f"X{st}", "full", "accumulating mma")
                    sim.expect("ACC", was, "accumulating mma")
                    sim.set(f"S{b}", "free"), sim.set("ACC", "acc")
                sim.pipe.append(run)
                sim.pipe.append(lambda st=st: (sim.set(f"X{st}", "free"), B[f"X_EMPTY{st}"].arrive()))
                if t == n - 1:
                    sim.pipe.append(lambda: (sim.set("ACC", "done"), B["ACC_FULL"].arrive()))
                g += 1
            n_it += 1

    def elements(w):
        g, n_it = 0, 0
        while True:
            n = yield from it.take(n_it)
            if n is None:
                return
            for _ in range(n):
                b = g & 1
                yield ("wait", f"S_FULL{b}", (g >> 1) & 1)
                sim.expect(f"S{b}", "s", f"element warps read S / dP of step {g}")
                if count_down(sim, f"S{b}_warps", 8):
                    sim.set(f"S{b}", "p")
                B[f"P_FULL{b}"].arrive()
                g += 1
            yield ("wait", "ACC_FULL", n_it & 1)
            sim.expect("ACC", "done", "output")
            if count_down(sim, "ACC_warps", 8):
                sim.set("ACC", "free")
            B["ACC_EMPTY"].arrive()
            n_it += 1

    return {"producer": producer(), "mma": mma(), **{f"elements{w}": elements(w) for w in range(8)}}


BWD_BARS = {"R_FULL": 1, "R_EMPTY": 1, "ACC_FULL": 1, "ACC_EMPTY": 8, **ITEM_BARS}
for _b in (0, 1):
    BWD_BARS.update({f"S_FULL{_b}": 1, f"P_FULL{_b}": 8})
for _st in range(X_STAGES):
    BWD_BARS.update({f"X_FULL{_st}": 1, f"X_EMPTY{_st}": 1})


@pytest.mark.parametrize("items", [[1], [2], [3], [4], [7], [12], [1, 1, 1, 1, 1], [2, 1, 3, 1], [5, 4, 3], [1, 8, 2, 1]], ids=str)
def test_backward_protocol_has_no_deadlock_or_buffer_hazard(items):
    for seed in range(100):
        sim = Sim(seed, BWD_BARS)
        sim.run(bwd_protocol(sim, items))
        assert all(v in ("free", 0) for v in sim.state.values()), sim.state


@pytest.mark.parametrize("parity", [lambda n: 1, lambda n: (n & 1) ^ 1], ids=["constant", "inverted"])
def test_the_model_checker_catches_a_wrong_parity(parity):
    """Sanity of the checker itself: a producer that waits for the resident tiles on the wrong phase is reported as a hazard or a deadlock."""
    failures = 0
    for seed in range(40):
        sim = Sim(seed, BWD_BARS)
        try:
            sim.run(bwd_protocol(sim, [3, 2, 4, 2], r_empty_parity=parity))
        except AssertionError:
            failures += 1
    assert failures > 0
