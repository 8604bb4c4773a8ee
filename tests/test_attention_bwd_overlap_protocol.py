"""Host restatement of the synchronisation of the attention backward with overlapping steps
(csrc/kernels/attention_bwd.cuh): S of the next step is formed over P as soon as dV has read it, dP of the next step over
dQ as soon as the softmax warps have read that.

  loader     Q(0) dO(0) Q(1), statistics 0 and 1; then per step it >= 1: do_empty(it-1) -> dO(it); q_empty(it-1) -> Q(it+1)
             and the statistics of it+1
  issuer     S(0) dP(0); per step: p_full -> dV, commit do_empty; q_full(it+1), do_empty -> S(it+1), commit s_full; ds_full -> dK,
             commit q_empty, dQ, commit dq_full; do_full(it+1), dq_read -> dP(it+1), commit dp_full
  softmax    per step: s_full, statistics -> P over S, p_full; dQ of the step before: dq_full -> read, dq_read, own_free of
             the step before that -> slabs, dqs_full; dp_full, shared_free of the step before -> dS, ds_full
  reducer    dqs_full -> reduce-adds; shared_free, own_free

Replayed with phase-parity barriers, a tensor pipe that promises an order only to products of one kind (one accumulator and
shape), whose commits arrive when everything issued before them has run, and random delays for loads, products, the reduce-adds and the softmax warps (two groups that finish at different
times): every product finds the operands of its own step, nothing is overwritten while something still reads it, and the walk ends for any number of steps.  Dropping one of the waits
must be noticed."""
import random

import pytest
from test_gemm_pair_protocol import Barrier

GROUPS = 2      # softmax warps modelled as two groups with independent timing


def simulate(iters, seed, drop=None):
    rng = random.Random(seed)
    bars = {n: Barrier() for n in ("q_full0", "q_full1", "q_empty0", "q_empty1", "do_full", "do_empty", "stat0", "stat1", "s_full",
                                   "dp_full", "dq_full", "shared_free", "own_free")}
    bars.update({n: Barrier(GROUPS) for n in ("p_full", "ds_full", "dq_read", "dqs_full")})
    holds = {k: None for k in ("Q0", "Q1", "dO", "dS", "tmS", "tmP", "own", "st0", "st1")}
    reads = {k: 0 for k in holds}
    pipe, inflight, tick, written = [], [], [0], {}

    def write(res, what):
        assert reads[res] == 0, f"{res} overwritten with {what} while {holds[res]} is still read"
        holds[res] = what

    def group_write(res, what):                       # the first softmax group to get there writes for all
        if written.get(res) != what:
            write(res, what)
            written[res] = what

    def wait(name, parity, key):
        return None if drop == key else ("wait", name, parity)

    def land(res, what, bar):
        def done():
            write(res, what)
            bars[bar].arrive()
        inflight.append((tick[0] + rng.choice((1, 20, 200)), done))

    def loader():
        def q(it):
            land(f"Q{it & 1}", ("Q", it), f"q_full{it & 1}")

        def stats(it):
            land(f"st{it & 1}", ("st", it), f"stat{it & 1}")
        q(0)
        land("dO", ("dO", 0), "do_full")
        stats(0)
        if iters > 1:
            q(1)
            stats(1)
        for it in range(1, iters):
            yield wait("do_empty", (it - 1) & 1, "do_empty")
            land("dO", ("dO", it), "do_full")
            if it + 1 == iters:
                break
            yield wait(f"q_empty{(it + 1) & 1}", ((it - 1) >> 1) & 1, "q_empty")
            q(it + 1)
            stats(it + 1)

    def issue(kind, it, operands, into, *commits):
        for r, _ in operands:
            reads[r] += 1
        pipe.append(("mma", kind, it, operands, into))
        pipe.extend(("commit", c) for c in commits)

    def issuer():
        s = lambda it: issue("S", it, [(f"Q{it & 1}", ("Q", it))], "tmS", "s_full")              # noqa: E731
        dp = lambda it: issue("dP", it, [("dO", ("dO", it))], "tmP", "dp_full")                  # noqa: E731
        yield ("wait", "q_full0", 0)
        s(0)
        yield ("wait", "do_full", 0)
        dp(0)
        for it in range(iters):
            ph, more = it & 1, it + 1 < iters
            yield wait("p_full", ph, "p_full")
            issue("dV", it, [("tmS", ("P", it)), ("dO", ("dO", it))], None, "do_empty")
            if more:
                yield wait(f"q_full{(it + 1) & 1}", ((it + 1) >> 1) & 1, "q_full")
                yield wait("do_empty", ph, "p_read")
                s(it + 1)
            yield wait("ds_full", ph, "ds_full")
            issue("dK", it, [("dS", ("dS", it)), (f"Q{it & 1}", ("Q", it))], None, f"q_empty{it & 1}")
            issue("dQ", it, [("dS", ("dS", it))], "tmP", "dq_full")
            if more:
                yield wait("do_full", (it + 1) & 1, "do_full")
                yield wait("dq_read", ph, "dq_read")
                dp(it + 1)

    def softmax(g):
        def dq_out(it):
            yield wait("dq_full", it & 1, "dq_full")
            assert holds["tmP"] == ("dQ", it)
            reads["tmP"] += 1
            yield ("work",)
            reads["tmP"] -= 1
            bars["dq_read"].arrive()
            if it > 0:
                yield wait("own_free", (it - 1) & 1, "own_free")
            group_write("own", ("dQ", it))
            group_write("dS", ("slab", it))
            bars["dqs_full"].arrive()

        for it in range(iters):
            ph = it & 1
            yield wait(f"stat{ph}", (it >> 1) & 1, "stat")
            yield wait("s_full", ph, "s_full")
            if holds["tmS"] != ("P", it):             # the other group may be ahead: its columns are its own
                assert holds["tmS"] == ("S", it), f"step {it} found {holds['tmS']}"
            assert holds[f"st{ph}"] == ("st", it)
            reads[f"st{ph}"] += 1
            yield ("work",)
            group_write("tmS", ("P", it))
            bars["p_full"].arrive()
            if it > 0:
                yield from dq_out(it - 1)
            yield wait("dp_full", ph, "dp_full")
            if it > 0:
                yield wait("shared_free", (it - 1) & 1, "shared_free")
            assert holds["tmP"] == ("dP", it)
            reads["tmP"] += 1
            yield ("work",)
            reads["tmP"] -= 1
            reads[f"st{ph}"] -= 1
            group_write("dS", ("dS", it))
            bars["ds_full"].arrive()
        yield from dq_out(iters - 1)

    def reducer():
        for it in range(iters):
            yield ("wait", "dqs_full", it & 1)
            assert holds["dS"] == ("slab", it) and holds["own"] == ("dQ", it)
            at = tick[0]
            for res, bar in (("dS", "shared_free"), ("own", "own_free")):
                reads[res] += 1

                def done(res=res, bar=bar):
                    reads[res] -= 1
                    bars[bar].arrive()
                at += rng.randint(1, 60)
                inflight.append((at, done))

    roles = {"loader": loader(), "issuer": issuer(), "reducer": reducer()}
    roles.update({f"softmax{g}": softmax(g) for g in range(GROUPS)})
    blocked, busy = {}, 0
    for _ in range(400000):
        tick[0] += 1
        for x in sorted((x for x in inflight if x[0] <= tick[0]), key=lambda x: x[0]):
            inflight.remove(x)
            x[1]()
        if pipe and tick[0] >= busy:
            products = [i for i, op in enumerate(pipe) if op[0] == "mma"][:2]
            swap = pipe[0][0] == "mma" and len(products) == 2 and pipe[products[1]][1] != pipe[0][1] and rng.random() < 0.3
            op = pipe.pop(products[1] if swap else 0)
            if op[0] == "commit":
                bars[op[1]].arrive()
            else:
                _, kind, it, operands, into = op
                for r, what in operands:
                    assert holds[r] == what, f"{kind} of step {it} found {holds[r]} in {r}"
                    reads[r] -= 1
                if into:
                    write(into, (kind, it))
                busy = tick[0] + rng.randint(1, 8)
        if not roles and not pipe and not inflight:
            return True
        if rng.random() < 0.4:
            continue
        order = list(roles)
        rng.shuffle(order)
        for name in order:
            if name in blocked:
                _, bar, parity = blocked[name]
                if not bars[bar].passed(parity):
                    continue
                del blocked[name]
            try:
                ev = next(roles[name])
            except StopIteration:
                del roles[name]
                break
            if ev and ev[0] == "wait" and not bars[ev[1]].passed(ev[2]):
                blocked[name] = ev
            break
    raise AssertionError(f"no progress: blocked {blocked}")


@pytest.mark.parametrize("iters", [1, 2, 3, 4, 9, 33])
def test_protocol_neither_deadlocks_nor_races(iters):
    for seed in range(40):
        assert simulate(iters, seed)


@pytest.mark.parametrize("drop", ["do_empty", "p_read", "q_empty", "p_full", "q_full", "ds_full", "do_full", "dq_read", "dq_full", "own_free",
                                  "stat", "s_full", "dp_full", "shared_free"])
def test_the_checker_sees_a_missing_wait(drop):
    with pytest.raises(AssertionError):
        for seed in range(300):
            simulate(12, seed, drop=drop)
