"""Products whose last tiles are divided along the reduction over CTA pairs: the division itself (restated here), and
the sums, which are exact in fp32 for small integers whatever their order."""
import pytest
import torch

SPLIT_MIN = 4


def _plan(lib, m, n, k, c_dtype=1, pairs=74):
    p = lib.ft_gemm_split_plan(m, n, k, c_dtype, pairs)
    return p & 0xffff, p >> 16 & 0xffff, p >> 32


def _begin(p, kt, tiles, pairs):
    """csrc/kernels/gemm2_kernel.cuh, SplitWork::begin"""
    b = p * tiles * kt // pairs
    r = b % kt
    return b - r if r < SPLIT_MIN else b + kt - r if kt - r < SPLIT_MIN else b


def _parts(pair, kt, tiles, pairs):
    """PairWork::part, the divided tiles only: (tile, first k-block, end) in the order of the work"""
    lo, hi = _begin(pair, kt, tiles, pairs), _begin(pair + 1, kt, tiles, pairs)
    mid = max(hi // kt * kt, lo)
    out = []
    if hi > mid:
        out.append((mid // kt, mid % kt, hi - mid // kt * kt))
    if mid > lo:
        out.append((lo // kt, lo % kt, kt))
    return out


def test_every_k_block_of_a_divided_tile_is_done_once_and_its_owner_finds_all_parts():
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    lib, divided = cuda_lib(), 0
    for pairs in (74, 66, 3, 2):
        for m in (129, 256, 1024, 2048, 3000, 4096, 16384):
            for n in (8, 64, 768, 1600, 4096, 6400, 11008, 50304):
                for k in (64, 200, 768, 1600, 2048, 11008, 50304):
                    tn, tiles, share = _plan(lib, m, n, k, 1, pairs)
                    if not tiles:
                        assert tn == lib.ft_gemm_tile_n(m, n, 1, pairs)
                        continue
                    divided += 1
                    kt = -(-k // 64)
                    assert tiles < share <= pairs and tiles == (-(-m // 256) * -(-n // tn)) % pairs
                    done = {}
                    for p in range(share):
                        parts = _parts(p, kt, tiles, share)
                        assert 1 <= len(parts) <= 2                     # two accumulators, one partial tile at most
                        assert sum(e != kt for _, _, e in parts) <= 1
                        for t, a, e in parts:
                            assert 0 <= a < e <= kt
                            done.setdefault(t, []).append((a, e, p))
                    for t in range(tiles):
                        runs = sorted(done[t])
                        assert runs[0][0] == 0 and runs[-1][1] == kt
                        assert all(x[1] == y[0] for x, y in zip(runs, runs[1:]))
                        owner = runs[-1][2]
                        assert [r[2] for r in runs] == list(range(owner - len(runs) + 1, owner + 1))
                        count = 0                                        # as the owner counts them
                        while count < owner and runs[-1][0] and _begin(owner - count, kt, tiles, share) > t * kt:
                            count += 1
                        assert count == len(runs) - 1
    assert divided > 100


# one tile for all pairs, several of a long reduction, a round and a bit, a ragged edge both ways
SHAPES = [(256, 64, 16384), (1024, 768, 12800), (3000, 1600, 6408), (2056, 2568, 8008), (300, 72, 20000)]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("mode", ["store16", "store32", "add16", "acc32"])
def test_products(m, n, k, a_mn, b_mn, mode):
    from flextrain_b200.ops.cuda_ops import gemm
    from flextrain_b200.ops.native import cuda_lib
    if a_mn and m % 8 or b_mn and n % 8:
        pytest.skip("rows of this operand are not 16-byte aligned")
    assert mode.endswith("32") or _plan(cuda_lib(), m, n, k)[1] > 0
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    # sums of at most 20000 products of up to 4: exact in fp32
    a, b = (torch.randint(-2, 3, (r, k), generator=gen, device="cuda").bfloat16() for r in (m, n))
    a_st, b_st = (t.t().contiguous() if mn else t for t, mn in ((a, a_mn), (b, b_mn)))
    dtype = torch.bfloat16 if mode.endswith("16") else torch.float32
    base = torch.randint(-50, 51, (m + 2, n), generator=gen, device="cuda").to(dtype)
    prod = a.double() @ b.double().T
    want = base.clone()
    want[1:-1] = (prod + (base[1:-1].double() if mode in ("add16", "acc32") else 0)).to(dtype)
    for _ in range(3):                                        # the workspace's memory comes back with old flags in it
        out = base.clone()
        if mode == "add16":
            gemm(a_st, a_mn, b_st, b_mn, m, n, k, out=out[1:-1], add=base[1:-1])
        else:
            gemm(a_st, a_mn, b_st, b_mn, m, n, k, out=out[1:-1], accumulate=mode == "acc32")
        torch.cuda.synchronize()
        assert cuda_lib().ft_gemm_error() == 0
        assert torch.equal(out, want)


@pytest.mark.gpu
def test_replayed_and_on_two_streams():
    """A captured product finds the flags of its last replay cleared; two streams have a workspace each."""
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, w = (torch.randint(-2, 3, s, generator=gen, device="cuda").bfloat16() for s in ((1024, 12800), (768, 12800)))
    bias = torch.randint(-2, 3, (768,), generator=gen, device="cuda").bfloat16()
    with torch.no_grad():
        want = (x.double() @ w.double().T + bias.double()).bfloat16()
        assert torch.equal(ops.linear_bias(x, w, bias), want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = ops.linear_bias(x, w, bias)
        for _ in range(3):
            y.zero_()
            graph.replay()
            assert torch.equal(y, want)
        side = [torch.cuda.Stream(), torch.cuda.Stream()]
        torch.cuda.synchronize()
        outs = []
        for i in range(6):
            with torch.cuda.stream(side[i % 2]):
                outs.append(ops.linear_bias(x, w, bias))
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs)
    assert cuda_lib().ft_gemm_error() == 0
