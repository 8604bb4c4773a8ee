"""Host replay of the products that are divided along the reduction (csrc/kernels/gemm2_kernel.cuh): the parts come
from the kernel's own division (``tile_walk.cuh``, compiled for the host), the order of what a warp does around a
flag from the source of ``split_store`` and ``split_wait``.

  issuer     per part of the pair's work: tmem_empty[it & 1] -> products, commit tmem_full[it & 1]
  epilogue   the parts that stay here: tmem_full -> partial sums to the workspace, flag, tmem_empty; then the tile the pair owns:
             the other pairs' flags -> their sums added in the order of the reduction, the tile stored, tmem_empty; then whole tiles

Every k-block must reach the result once and in order, no accumulator be overwritten before it is read, and the walk end
with any number of pairs on the chip, as long as they start in the order of their numbers.  Lanes carry vector clocks: a
partial sum may be read by a lane only where the writer's store is ordered before it."""
import os
import random
import re

import pytest
from test_gemm_pair_protocol import Barrier
from test_gemm_split_gpu import _plan
from test_tile_walk import ask, build_walk

KERNEL = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc", "kernels", "gemm2_kernel.cuh")
LANES = 3                                             # the one that handles the flag and two others


def steps(function):
    """What orders memory in a device function of the kernel, as it stands in the source."""
    body = re.search(r"\b%s\(.*?\n}\n" % function, open(KERNEL).read(), re.S).group(0)
    names = {"__threadfence()": "fence", "__syncwarp()": "warp", "st.release": "release", "ld.acquire": "acquire",
             "out[(c * 8": "write", "__shfl_sync": "verdict"}
    found = sorted((m.start(), what) for text, what in names.items() for m in re.finditer(re.escape(text), body))
    return [what for _, what in found]


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    return build_walk(tmp_path_factory.mktemp("walk"))


def merge(a, b):
    for k, v in b.items():
        a[k] = max(a.get(k, 0), v)


def simulate(parts, whole, kt, resident, seed, store, wait, order=None, drop=None):
    """``parts[p]``: the work of pair p, (tile, first k-block, end) each; the last ``len - ...`` of them whole tiles."""
    rng = random.Random(seed)
    pairs = len(parts)
    bars = {(p, n, a): Barrier() for p in range(pairs) for n in ("full", "empty") for a in (0, 1)}
    acc, reading = {}, {}                             # (pair, accumulator) -> contents; being read
    sums, flags, result = {}, {}, {}
    clock = {(p, lane): {(p, lane): 1} for p in range(pairs) for lane in range(LANES)}

    def tick(p, lane):
        clock[p, lane][p, lane] = clock[p, lane].get((p, lane), 0) + 1

    def warp(p):                                      # a warp barrier orders every lane after every other
        top = {}
        for lane in range(LANES):
            merge(top, clock[p, lane])
        for lane in range(LANES):
            merge(clock[p, lane], top)
            tick(p, lane)

    def issuer(p):
        for it, (tile, a, e) in enumerate(parts[p]):
            if drop != "tmem_empty":
                yield lambda it=it: bars[p, "empty", it & 1].passed((it >> 1 & 1) ^ 1)
            yield None
            assert not reading.get((p, it & 1)), f"accumulator {it & 1} of pair {p} overwritten while it is read"
            acc[p, it & 1] = (tile, list(range(a, e)))
            reading[p, it & 1] = True
            bars[p, "full", it & 1].arrive()

    def read(p, it):
        return acc[p, it & 1]

    def leave(p, it):
        reading[p, it & 1] = False
        bars[p, "empty", it & 1].arrive()

    def epilogue(p):
        owned, it = None, 0
        for it, (tile, a, e) in enumerate(parts[p]):
            yield lambda it=it: bars[p, "full", it & 1].passed(it >> 1 & 1)
            got = read(p, it)
            assert got[0] == tile
            blocks = got[1]
            if e != kt:                               # stays in the workspace
                for what in store:
                    if what == "write":
                        for lane in range(LANES):
                            tick(p, lane)
                            sums[p, lane] = (tile, blocks, dict(clock[p, lane]))
                        yield None
                    elif what == "warp":
                        warp(p)
                    elif what == "release":
                        flags[p] = (tile, dict(clock[p, 0]))
                        tick(p, 0)
                leave(p, it)
                continue
            if a != 0:                                # owned: the pairs before this one hold the rest
                first = a
                others = []
                while first:
                    q = p - len(others) - 1
                    others.append(q)
                    first = next(x for t, x, y in parts[q] if t == tile)
                assert owned is None
                owned, before = tile, []
                for q in sorted(others):
                    for what in wait:
                        if what == "acquire":
                            yield lambda q=q: flags.get(q) is not None
                            assert flags[q][0] == tile
                            merge(clock[p, 0], flags[q][1])
                            flags[q] = None           # cleared for the next launch
                            tick(p, 0)
                        elif what == "warp":
                            warp(p)
                    for lane in range(LANES):
                        t, b, then = sums[q, lane]
                        assert t == tile
                        assert clock[p, lane].get((q, lane), 0) >= then[q, lane], f"lane {lane} reads unordered sums"
                    before += sums[q, 0][1]
                blocks = before + blocks
            yield None
            assert blocks == list(range(kt)), f"tile {tile}: {blocks}"
            assert tile not in result
            result[tile] = p
            leave(p, it)

    waiting = list(order or range(pairs))
    roles, blocked = {}, {}
    for _ in range(400000):
        while waiting and len({p for p, _ in roles}) < resident:
            p = waiting.pop(0)
            roles[p, "mma"], roles[p, "epi"] = issuer(p), epilogue(p)
        if not roles:
            break
        ready = [k for k in roles if k not in blocked or blocked[k]()]
        if not ready:
            raise AssertionError(f"no progress: {sorted(roles)}")
        key = rng.choice(ready)
        blocked.pop(key, None)
        try:
            cond = next(roles[key])
        except StopIteration:
            del roles[key]
            continue
        if cond is not None:
            blocked[key] = cond
    assert sorted(result) == list(range(whole))
    assert not any(flags.values()), "a flag that nobody cleared"


def divisions(walk, pairs, count, seed):
    """Work of every pair for ``count`` products that the library's own rule divides."""
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    rng, found = random.Random(seed), []
    while len(found) < count:
        m, n, k = rng.randint(129, 4000), 8 * rng.randint(1, 500), rng.randint(4000, 60000)
        width, tiles, share = _plan(cuda_lib(), m, n, k, 1, pairs)
        if tiles:
            found.append((-(-m // 256) * -(-n // width), -(-k // 64), tiles, share))
    used = [max(share, min(total, pairs)) for total, _, _, share in found]
    lines = ask(walk, [f"parts {u} {total} {kt} {tiles} {share}" for u, (total, kt, tiles, share) in zip(used, found)])
    for u, (total, kt, _, _) in zip(used, found):
        yield [lines.pop(0) for _ in range(u)], total, kt


def test_sums_arrive_whole_and_in_order(walk):
    store, wait = steps("split_store"), steps("split_wait")
    assert "write" in store and "release" in store and "acquire" in wait
    for pairs in (3, 6, 11):
        for i, (parts, total, kt) in enumerate(divisions(walk, pairs, 12, pairs)):
            for resident in (1, 2, pairs):            # pairs that find room at a time, started in order
                simulate(parts, total, kt, resident, i, store, wait)


def test_the_replay_sees_what_is_left_out(walk):
    store, wait = steps("split_store"), steps("split_wait")
    work = list(divisions(walk, 6, 12, 1))
    for changed in (dict(wait=[w for w in wait if w != "warp"]), dict(store=[s for s in store if s != "warp"]),
                    dict(drop="tmem_empty")):
        with pytest.raises(AssertionError):
            for i, (parts, total, kt) in enumerate(work * 20):
                simulate(parts, total, kt, 6, i, **{**dict(store=store, wait=wait), **changed})
    with pytest.raises(AssertionError, match="no progress"):      # what the order of the launch is needed for
        for i, (parts, total, kt) in enumerate(work):
            simulate(parts, total, kt, 1, i, store, wait, order=range(len(parts) - 1, -1, -1))
