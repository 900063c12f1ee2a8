"""Model check of the barrier protocol of the attention forward with output warps of its own (csrc/attn_fwd_tcgen05.cu), on the simulator of
test_attention_pipeline_protocol_cpu.py: the waits, arrivals and commits of every role of a CTA in the kernel's order."""
import pytest
from test_attention_pipeline_protocol_cpu import BOTH, ONE, SECOND, STAGES, Items, Sim, count_down, load

READERS = 13                       # of an item: MMA, 8 softmax warps, 4 output warps


def bars():
    b = {"IT_FULL0": 1, "IT_FULL1": 1, "IT_EMPTY0": READERS, "IT_EMPTY1": READERS, "CLC_FULL": 1}
    for t in (0, 1):
        b.update({f"Q_FULL{t}": 1, f"Q_EMPTY{t}": 1, f"S_FULL{t}": 1, f"P_FULL{t}": 8, f"O_FULL{t}": 1, f"L_FULL{t}": 4, f"L_EMPTY{t}": 4, **{f"A_FULL{t}{q}": 1 for q in range(4)}})
    for i in range(STAGES):
        b.update({f"KV_FULL{i}": 1, f"KV_EMPTY{i}": 1})
    return b


def protocol(sim, items, mistake=None):
    """An item is the list of its key tiles, each (taken by query tile 0, taken by query tile 1).  mistake: "scale" (the output warps arrive for a tile before they
    have scaled O), "order" (they take all of tile 0's key tiles before tile 1's)."""
    B = sim.bars
    it = Items(sim, items, READERS)

    def producer():
        kvc, qc, idx = 0, [0, 0], 0
        it.request()
        while idx is not None:
            walk = items[idx]
            yield from it.publish(walk)

            def load_q(t):
                if any(k[t] for k in walk):
                    yield ("wait", f"Q_EMPTY{t}", (qc[t] & 1) ^ 1)
                    qc[t] += 1
                    load(sim, f"Q{t}", f"Q_FULL{t}", 2, "Q load")

            def load_kv():
                nonlocal kvc
                st = kvc % STAGES
                yield ("wait", f"KV_EMPTY{st}", ((kvc // STAGES) & 1) ^ 1)
                kvc += 1
                load(sim, f"KV{st}", f"KV_FULL{st}", 2, "K / V load")
            yield from load_q(0)
            yield from load_kv()
            yield from load_q(1)
            yield from load_kv()
            for _ in walk[1:]:
                yield from load_kv()
                yield from load_kv()
            idx = yield from it.next()
            if idx is not None:
                it.request()
        yield from it.publish(None)

    def mma():
        kvc, qc, pc, n_it = 0, [0, 0], [0, 0], 0
        while True:
            walk = yield from it.take(n_it)
            n_it += 1
            if walk is None:
                return
            s_open, o_open = [False, False], [False, False]
            last = [max((k for k, x in enumerate(walk) if x[t]), default=-1) for t in range(2)]

            def pass_kv(c):
                yield ("wait", f"KV_FULL{c % STAGES}", (c // STAGES) & 1)
                return c % STAGES

            def free_kv(st):
                sim.pipe.append(lambda: (sim.set(f"KV{st}", "free"), B[f"KV_EMPTY{st}"].arrive()))

            def issue_s(t, k, st):
                if not s_open[t]:
                    yield ("wait", f"Q_FULL{t}", qc[t] & 1)
                    qc[t] += 1
                    s_open[t] = True

                def run():
                    sim.expect(f"Q{t}", "full", "S mma"), sim.expect(f"KV{st}", "full", "S mma"), sim.expect(f"S{t}", "free", "S mma")
                    sim.set(f"S{t}", "s")
                sim.pipe.append(run)
                sim.pipe.append(lambda: B[f"S_FULL{t}"].arrive())
                if k == last[t]:
                    sim.pipe.append(lambda: (sim.set(f"Q{t}", "free"), B[f"Q_EMPTY{t}"].arrive()))

            def issue_pv(t, k, st):
                yield ("wait", f"P_FULL{t}", pc[t] & 1)
                pc[t] += 1
                was, o_open[t] = "acc" if o_open[t] else "free", True
                sim.state[f"PV{t}"] = sim.state.get(f"PV{t}", 0) + 1           # issued and not retired

                def run():
                    sim.expect(f"S{t}", "p", "PV mma"), sim.expect(f"KV{st}", "full", "PV mma"), sim.expect(f"O{t}", was, "PV mma")
                    sim.set(f"S{t}", "free"), sim.set(f"O{t}", "acc")
                    sim.state[f"PV{t}"] -= 1
                sim.pipe.append(run)
                if k == last[t]:
                    sim.pipe.append(lambda: B[f"O_FULL{t}"].arrive())
            st = yield from pass_kv(kvc)
            for t in range(2):
                if walk[0][t]:
                    yield from issue_s(t, 0, st)
            free_kv(st)
            for k in range(len(walk)):
                sv, sk = (yield from pass_kv(kvc + 2 * k + 1)), None
                for t in range(2):
                    if walk[k][t]:
                        yield from issue_pv(t, k, sv)
                    if k + 1 < len(walk):
                        if sk is None:
                            sk = yield from pass_kv(kvc + 2 * k + 2)
                        if walk[k + 1][t]:
                            yield from issue_s(t, k + 1, sk)
                    if t == 1:
                        free_kv(sv)
                if sk is not None:
                    free_kv(sk)
            kvc += 2 * len(walk)

    def softmax(w):
        t, quad, sc, n_it, n_l = w >> 2, w & 3, 0, 0, 0
        while True:
            walk = yield from it.take(n_it)
            n_it += 1
            if walk is None:
                return
            n_tiles = sum(k[t] for k in walk)
            if n_tiles == 0:
                continue
            for k in range(n_tiles):
                yield ("wait", f"S_FULL{t}", sc & 1)
                sc += 1
                sim.expect(f"S{t}", "s", "softmax reads S")
                if k > 0:
                    sim.expect(f"alpha{t}{quad}", "free", "factors are written")
                    sim.set(f"alpha{t}{quad}", "full")
                    B[f"A_FULL{t}{quad}"].arrive()
                    yield ("wait", f"S_FULL{t}", (sc - 1) & 1)                  # passed already: the others may run while the weights are formed
                if count_down(sim, f"S{t}_warps", 4):
                    sim.set(f"S{t}", "p")
                B[f"P_FULL{t}"].arrive()
            yield ("wait", f"L_EMPTY{t}", (n_l & 1) ^ 1)
            n_l += 1
            sim.expect(f"l{t}{quad}", "free", "denominators are written")
            sim.set(f"l{t}{quad}", "full")
            B[f"L_FULL{t}"].arrive()

    def output(quad):
        ac, oc, n_it = [0, 0], [0, 0], 0
        for t in range(2):
            B[f"P_FULL{t}"].arrive()
        while True:
            walk = yield from it.take(n_it)
            n_it += 1
            if walk is None:
                return
            opened = [False, False]
            order = [(k, t) for k in range(len(walk)) for t in range(2)] if mistake != "order" else [(k, t) for t in range(2) for k in range(len(walk))]
            for k, t in order:
                if not walk[k][t]:
                    continue
                if opened[t]:
                    if mistake != "scale":
                        yield ("wait", f"A_FULL{t}{quad}", ac[t] & 1)
                    ac[t] += 1
                    sim.expect(f"alpha{t}{quad}", "full", "factors are read")
                    assert sim.state[f"PV{t}"] == 0, "O is scaled with a product in flight"
                    sim.expect(f"O{t}", "acc", "O is scaled")
                    sim.set(f"alpha{t}{quad}", "free")
                    B[f"P_FULL{t}"].arrive()
                opened[t] = True
            for t in range(2):
                if not any(k[t] for k in walk):
                    continue
                yield ("wait", f"L_FULL{t}", oc[t] & 1)
                sim.expect(f"l{t}{quad}", "full", "denominators are read")
                sim.set(f"l{t}{quad}", "free")
                B[f"L_EMPTY{t}"].arrive()
                yield ("wait", f"O_FULL{t}", oc[t] & 1)
                oc[t] += 1
                sim.expect(f"O{t}", "acc", "output")
                assert sim.state[f"PV{t}"] == 0, "output with a product in flight"
                if count_down(sim, f"O{t}_warps", 4):
                    sim.set(f"O{t}", "free")
                B[f"P_FULL{t}"].arrive()

    return {"producer": producer(), "mma": mma(), **{f"softmax{w}": softmax(w) for w in range(8)}, **{f"output{q}": output(q) for q in range(4)}}


WALKS = [[[BOTH]], [[ONE]], [[BOTH] * 3 + [ONE]], [[ONE]] * 5, [[BOTH]] * 5, [[BOTH] * 2 + [ONE], [ONE], [BOTH] * 5, [ONE] * 3],
         [[SECOND] * 2 + [BOTH] * 2 + [ONE], [BOTH, SECOND, BOTH, ONE], [ONE]], [[BOTH] * 9, [BOTH] * 2 + [ONE], [BOTH] * 4]]


@pytest.mark.parametrize("items", WALKS, ids=lambda x: "-".join(str(len(w)) for w in x))
def test_no_deadlock_or_buffer_hazard(items):
    for seed in range(60):
        sim = Sim(seed, bars())
        sim.run(protocol(sim, items))
        assert all(v in ("free", 0) for v in sim.state.values()), sim.state


@pytest.mark.parametrize("mistake", ["scale", "order"])
def test_the_model_finds_planted_mistakes(mistake):
    failures = 0
    for seed in range(20):
        sim = Sim(seed, bars())
        try:
            sim.run(protocol(sim, [[SECOND] * 2 + [BOTH] * 2 + [ONE], [BOTH] * 3], mistake))
        except AssertionError:
            failures += 1
    assert failures > 0
