"""Bias and GELU over rows that are no multiple of what a block takes, narrower than a warp and wider, with one row and
with four a thread; against float64.  A 16-bit result is one rounding (2^-9 of it) of an fp32 value whose exponential and quotient are good to a few
2^-22; 2^-8 leaves room for both."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n", [(1, 8), (31, 248), (33, 264), (2048, 3072), (70001, 24), (31001, 40),
                                    (65535 * 32 + 5, 8)])
def test_forward_and_backward(rows, n):
    from flextrain_b200.ops import cuda_ops as ops
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x, dy = (torch.randn(rows, n, generator=gen, device="cuda").mul_(3).bfloat16() for _ in range(2))
    b = torch.randn(n, generator=gen, device="cuda").bfloat16()
    x.requires_grad_(), b.requires_grad_()
    y = ops.bias_gelu(x, b)
    y.backward(dy)
    u = (x.detach().float() + b.detach().float()).double().requires_grad_()
    want = torch.nn.functional.gelu(u, approximate="tanh")
    want.backward(dy.double())
    near = lambda a, w: ((a.double() - w).abs() <= 2 ** -8 * w.abs() + 1e-5 * dy.abs().max()).all()        # noqa: E731
    assert near(y.detach(), want.detach()) and near(x.grad, u.grad)
    total = u.grad.sum(0)
    assert ((b.grad.double() - total).abs() <= 2 ** -8 * total.abs() + 2 ** -8 * rows ** 0.5).all()
    with torch.no_grad():
        assert torch.equal(ops.bias_add(x.detach().clone(), b), (x.float() + b.float()).bfloat16())


def test_values_of_any_size():
    """The derivative is 1 or 0 far from the origin, whatever its polynomial overflows to; NaN stays NaN.  bf16 holds
    values up to 3e38, and every 16-bit number is tried."""
    from flextrain_b200.ops import cuda_ops as ops
    for dtype in (torch.bfloat16, torch.float16):
        x = torch.arange(-32768, 32768, device="cuda").to(torch.int16).view(dtype).reshape(-1, 8).clone().requires_grad_()
        b = torch.zeros(8, dtype=dtype, device="cuda", requires_grad=True)
        y = ops.bias_gelu(x, b)
        y.backward(torch.ones_like(y))
        u = x.detach().double()
        finite, far = u.isfinite(), u.abs() > 16
        held = u.clamp(-16, 16).requires_grad_()
        want = torch.nn.functional.gelu(held, approximate="tanh")
        want.sum().backward()
        value = torch.where(far, u.clamp(min=0), want.detach())
        near = lambda a, w: ((a.double() - w).abs() <= 2 ** -8 * w.abs() + 1e-5)[finite].all()             # noqa: E731
        assert near(y.detach(), value) and near(x.grad, held.grad)
        assert torch.equal(x.grad[far & finite], (u > 0).to(dtype)[far & finite])
        assert y.isnan()[u.isnan()].all() and x.grad.isnan()[u.isnan()].all()
