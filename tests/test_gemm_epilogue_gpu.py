"""The 16-bit GEMM epilogue by way of shared memory: both kernels (up to 128 rows and above), chunks of 32 columns cut
by the matrix's edge, rows cut by it, outputs and addends that are columns of wider matrices, and the shapes that take
the element path.  Small integers: every sum is exact in fp32, the result is the exact one rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 33, 128, 129, 500, 777])
@pytest.mark.parametrize("n", [8, 24, 32, 40, 72, 256, 264, 1000, 1001])
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
