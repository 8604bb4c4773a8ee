"""The CTA-pair GEMM with tiles narrower than 256 columns: the rule that picks the width (restated here and
compared with the library's), and products at shapes that pick each width, in the operand layouts of forward, data and
weight gradients."""
import pytest
import torch


def pair_tile_n(m, n, pairs=74):
    """csrc/kernels/gemm_tcgen05.cu, 16-bit results"""
    mt = -(-m // 256)
    cost = lambda bn: -(-mt * -(-n // bn) // pairs) * (bn + 128)                   # noqa: E731
    return min((256, 128, 64), key=lambda bn: (cost(bn), -bn))


SHAPES = {(300, 264): 64, (257, 8): 64, (2000, 1032): 128, (1900, 768): 128, (1000, 768): 64, (2000, 2304): 256, (3000, 1600): 256}


@pytest.mark.parametrize("shape,width", SHAPES.items())
def test_the_shapes_below_cover_every_width(shape, width):
    assert pair_tile_n(*shape) == width


def test_the_rule_is_the_librarys():
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    lib = cuda_lib()
    for m in (129, 256, 257, 1000, 2048, 3000, 4096, 32768):
        for n in (8, 64, 264, 768, 1032, 1600, 2304, 4096, 6400, 13824, 50304):
            for pairs in (74, 66, 1):
                assert lib.ft_gemm_tile_n(m, n, 1, pairs) == pair_tile_n(m, n, pairs)
                assert lib.ft_gemm_tile_n(m, n, 0, pairs) == 256      # fp32 results


@pytest.mark.parametrize("m", [129, 256, 2048, 4096, 32768])
@pytest.mark.parametrize("n", [64, 768, 1600, 4096, 13824, 50304])
def test_a_narrow_tile_never_costs_rounds_it_does_not_win_back(m, n):
    mt, bn = -(-m // 256), pair_tile_n(m, n)
    rounds = lambda b: -(-mt * -(-n // b) // 74)                                  # noqa: E731
    assert rounds(bn) * bn <= rounds(256) * 256


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("mode", ["store16", "store32", "add16", "acc32"])
def test_products(m, n, a_mn, b_mn, mode):
    from flextrain_b200.ops.cuda_ops import gemm
    from flextrain_b200.ops.native import cuda_lib
    k = 200                                               # three k-blocks and a part of one
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    # small integers: every sum is exact in fp32, a 16-bit result is the exact one rounded once
    a, b = (torch.randint(-2, 3, (r, k), generator=gen, device="cuda").bfloat16() for r in (m, n))
    a_st, b_st = (t.t().contiguous() if mn else t for t, mn in ((a, a_mn), (b, b_mn)))
    if a_mn and m % 8 or b_mn and n % 8:
        pytest.skip("rows of this operand are not 16-byte aligned")
    dtype = torch.bfloat16 if mode.endswith("16") else torch.float32
    base = torch.randint(-50, 51, (m + 2, n), generator=gen, device="cuda").to(dtype)
    out, want = base.clone(), base.clone()
    prod = a.double() @ b.double().T
    if mode == "add16":
        gemm(a_st, a_mn, b_st, b_mn, m, n, k, out=out[1:-1], add=base[1:-1])
    else:
        gemm(a_st, a_mn, b_st, b_mn, m, n, k, out=out[1:-1], accumulate=mode == "acc32")
    want[1:-1] = (prod + (base[1:-1].double() if mode in ("add16", "acc32") else 0)).to(dtype)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    assert torch.equal(out, want)
