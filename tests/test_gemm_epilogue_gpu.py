"""The 16-bit GEMM epilogue by way of shared memory and the one from registers: both kernels (up to 128 rows and above),
chunks of 32 columns cut by the matrix's edge inside and between its units of eight, rows cut by it, outputs and addends that
are columns of wider matrices, and the shapes that take the element path.  Small integers: every sum is exact in fp32,
the result is the exact one rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 33, 128, 129, 500, 777])
@pytest.mark.parametrize("n", [8, 24, 31, 32, 33, 40, 72, 256, 264, 1000, 1001, 1007])
@pytest.mark.parametrize("mode", ["store", "add", "accumulate", "bias", "bias_add"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_outputs(m, n, mode, dtype):
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    k = 136
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    ints = lambda hi, *s: torch.randint(-hi, hi + 1, s, generator=gen, device="cuda").to(dtype)      # noqa: E731
    a, b, bias = ints(2, m, k), ints(2, n, k), ints(9, n)
    wide = lambda: ints(50, m + 2, n + 16 + (8 - n % 8) % 8)                                         # noqa: E731
    prod = a.double() @ b.double().T
    held, addend = wide(), wide()
    cols = slice(8, 8 + n)
    out = held.clone()
    if mode.startswith("bias"):
        if n % 8:
            pytest.skip("the bias needs columns in eights")
        res = addend[1:-1, cols] if mode == "bias_add" else None
        out[1:-1, cols] = ops.linear_bias(a, b, bias, res)
        want = prod + bias.double() + (0 if res is None else res.double())
    elif mode == "add":
        ops.gemm(a, False, b, False, m, n, k, out=out[1:-1, cols], add=addend[1:-1, cols])
        want = prod + addend[1:-1, cols].double()
    else:
        ops.gemm(a, False, b, False, m, n, k, out=out[1:-1, cols], accumulate=mode == "accumulate")
        want = prod + (held[1:-1, cols].double() if mode == "accumulate" else 0)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    expect = held.clone()
    expect[1:-1, cols] = want.to(dtype)
    assert torch.equal(out, expect)


def _rule(m, n, k, add=0, bias=0, c_dtype=1):
    from flextrain_b200.ops.native import cuda_lib
    return bool(cuda_lib().ft_gemm_staged(m, n, k, c_dtype, add, bias, 74))


def test_the_rule():
    assert all(_rule(m, n, 64, add=1) for m in (1, 128, 129, 4096) for n in (32, 40, 4096))
    assert not _rule(4096, 33, 64, add=1)
    assert not any(_rule(m, n, 4096, a, b, 0) for m in (1, 4096) for n in (32, 4096) for a in (0, 1) for b in (0, 1))
    assert not any(_rule(m, n, 768, add=a, bias=b) for m in (1, 4096) for n in (8, 24) for a in (0, 1) for b in (0, 1))
    assert not any(_rule(m, n, 64, bias=b) for m in (1, 32) for n in (32, 40, 4096) for b in (0, 1))
    assert _rule(33, 64, 64, bias=1) and not _rule(128, 4096, 1024) and not _rule(128, 40, 64)
    assert not _rule(4096, 4096, 704) and _rule(4096, 4096, 768) and not _rule(2048, 2048, 4096)
    assert _rule(4096, 4104, 64) and _rule(4096, 4096, 64, bias=1) and not _rule(4096, 4097, 4096)


# several tiles for every pair, whole (two accumulators, slots that the next tile's addends fill) on both epilogues
@pytest.mark.parametrize("m,n,k", [(6000, 2568, 64), (4096, 2560, 64), (4096, 2560, 776), (2100, 3001, 64), (257, 777, 64),
                                   (129, 248, 64), (128, 256, 64), (40, 1000, 64), (1, 8, 64)])
@pytest.mark.parametrize("mode", ["store", "add", "accumulate", "bias", "bias_add"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_several_tiles(m, n, k, mode, dtype):
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    # integers up to 3, at most 776 products of them: exact in fp32
    ints = lambda hi, *s: torch.randint(-hi, hi + 1, s, generator=gen, device="cuda")                # noqa: E731
    a, b, bias = ints(3, m, k).bfloat16(), ints(3, n, k).bfloat16(), ints(9, n).bfloat16()
    ld = (n + 7) // 8 * 8                                 # rows stay aligned where n is odd
    held, addend = ints(100, m + 2, ld).to(dtype), ints(100, m + 2, ld).to(dtype)
    prod, at, out = a.double() @ b.double().T, (slice(1, -1), slice(0, n)), held.clone()
    if mode.startswith("bias"):
        if n % 8 or dtype == torch.float32:
            pytest.skip("no bias in this form")
        res = addend[at] if mode == "bias_add" else None
        out[at] = ops.linear_bias(a, b, bias, res)
        want = prod + bias.double() + (0 if res is None else res.double())
    elif mode == "add":
        ops.gemm(a, False, b, False, m, n, k, out=out[at], add=addend[at])
        want = prod + addend[at].double()
    else:
        ops.gemm(a, False, b, False, m, n, k, out=out[at], accumulate=mode == "accumulate")
        want = prod + (held[at].double() if mode == "accumulate" else 0)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    expect = held.clone()
    expect[at] = want.to(dtype)
    assert torch.equal(out, expect)                       # the rows around the output and the columns behind it too


# K on both sides of the line between the epilogues of the activation alone
@pytest.mark.parametrize("k", [512, 520])
def test_gate_alone(k):
    """Projections that are exact in fp32 (multiples of 1/16): what is left are the exponential, the quotient and one
    rounding, as in ``test_gate``."""
    from flextrain_b200.ops import cuda_ops as ops
    gen = torch.Generator(device="cuda").manual_seed(k)
    x, w = (torch.randint(-1, 2, s, generator=gen, device="cuda").bfloat16() for s in ((500, k), (768, k)))
    x = x / 16
    gu = x.double() @ w.double().T
    want = torch.nn.functional.silu(gu[:, :384]) * gu[:, 384:]
    with torch.no_grad():
        act = ops.linear_swiglu(x, w)
    assert ((act.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("rows,f", [(129, 128), (500, 384)])
@pytest.mark.parametrize("keep", [False, True])
def test_gate(rows, f, keep):
    """act and the kept projections of the gated product, at rows that are no multiple of anything; the activation
    against fp32 (its exponential and quotient are within a few 2^-22, the result rounded to bf16: 2^-9)."""
    from flextrain_b200.ops import cuda_ops as ops
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x, w = (torch.randn(*s, generator=gen, device="cuda").bfloat16() for s in ((rows, 200), (2 * f, 200)))
    x = (x * 0.2).requires_grad_(keep)
    act = ops.linear_swiglu(x, w)
    gu = x.detach().double() @ w.double().T
    want = torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]
    assert ((act.detach().double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()
    if keep:
        dy = torch.randn(rows, f, generator=gen, device="cuda").bfloat16()
        act.backward(dy)
        g = gu.to(torch.bfloat16).double().requires_grad_()          # the projections as they are kept
        (torch.nn.functional.silu(g[:, :f]) * g[:, f:]).backward(dy.double())
        dgu = g.grad @ w.double()
        assert (x.grad.double() - dgu).norm() < 0.01 * dgu.norm()
