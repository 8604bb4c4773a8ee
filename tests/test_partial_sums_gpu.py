"""Column sums of the per-CTA partial rows (bias and gain gradients): widths around the 32-column CTA,
row counts that leave one partial row, fewer than 32 of them and all."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 40, 256, 1608])
@pytest.mark.parametrize("rows", [1, 9, 300, 5000])
def test_bias_and_gain_gradients_are_exact_sums(rows, n):
    from flextrain_b200.ops.cuda_ops import bias_add, layernorm
    gen = torch.Generator(device="cuda").manual_seed(rows + n)
    # small integers: every partial sum is exact in fp32, the gradient is the sum rounded once
    dy = torch.randint(-4, 5, (rows, n), generator=gen, device="cuda").to(torch.bfloat16)
    want = dy.double().sum(0).to(torch.bfloat16)
    bias = torch.zeros(n, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    x = torch.randn(rows, n, generator=gen, device="cuda").bfloat16()
    bias_add(x.clone(), bias).backward(dy)
    assert torch.equal(bias.grad, want)
    w = torch.ones(n, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    b = torch.zeros(n, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    layernorm(x, w, b, 1e-5).backward(dy)
    assert torch.equal(b.grad, want)
    xh = torch.nn.functional.layer_norm(x.double(), (n,), eps=1e-5)
    err = (w.grad.double() - (dy.double() * xh).sum(0)).norm() / (dy.double() * xh).sum(0).norm()
    assert err < 0.01                                    # one bf16 rounding: 2^-9 per element at most
