"""Bias and residual in the GEMM epilogue, LayerNorm with the residual add: results and every gradient
against fp64, at row and column counts around the kernels' tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# every result is one fp32 sum rounded to the type: 2^-9 (bf16) or 2^-12 (fp16) per element, and fp32
# sums of up to 1000 terms below that; inputs to the backward are the same on both sides
TOL = {torch.bfloat16: 3e-3, torch.float16: 4e-4}


def _err(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("rows,n", [(1, 8), (128, 264), (129, 256), (300, 1000)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("residual", [False, True])
def test_linear_bias(rows, n, dtype, residual):
    from flextrain_b200.ops import functional as F
    k = 72
    gen = torch.Generator(device="cuda").manual_seed(rows + n)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)      # noqa: E731
    ins = [rand(rows, k), rand(n, k), rand(n)] + ([rand(rows, n)] if residual else [])
    ins = [t.requires_grad_() for t in ins]
    dy = rand(rows, n)
    y = F.linear_bias_add(*ins) if residual else F.linear_bias(*ins)
    y.backward(dy)
    ref = [t.detach().double().requires_grad_() for t in ins]
    want = torch.nn.functional.linear(*ref[:3]) + (ref[3] if residual else 0)
    want.backward(dy.double())
    assert _err(y, want) < TOL[dtype]
    for a, b in zip(ins, ref):
        assert _err(a.grad, b.grad) < TOL[dtype]


def test_a_bias_the_kernels_cannot_read_is_refused():
    from flextrain_b200.ops import functional as F
    x = torch.randn(4, 64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError):                     # a width that is no multiple of 8
        F.linear_bias(x, torch.randn(12, 64, device="cuda").bfloat16(), torch.zeros(12, device="cuda").bfloat16())
    with pytest.raises(RuntimeError):                     # a bias that starts off a 16-byte boundary
        F.linear_bias(x, torch.randn(16, 64, device="cuda").bfloat16(), torch.zeros(17, device="cuda").bfloat16()[1:])
    with pytest.raises(ValueError):
        F.linear_bias(x, torch.randn(16, 64, device="cuda").bfloat16(), torch.zeros(8, device="cuda").bfloat16())


@pytest.mark.parametrize("rows,h", [(1, 64), (37, 768), (130, 5128)])
@pytest.mark.parametrize("both", [False, True])
def test_add_layernorm(rows, h, both):
    from flextrain_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x, r, ds, dy = (torch.randint(-8, 9, (rows, h), generator=gen, device="cuda").div(4).bfloat16() for _ in range(4))
    w, b = (torch.randn(h, generator=gen, device="cuda").bfloat16() for _ in range(2))
    ins = [t.requires_grad_() for t in (x, r, w, b)]
    s, y = F.add_layernorm(*ins, 1e-5)
    ref = [t.detach().double().requires_grad_() for t in ins]
    s64 = ref[0] + ref[1]                                 # quarters: exact in bf16
    y64 = torch.nn.functional.layer_norm(s64, (h,), ref[2], ref[3], 1e-5)
    if both:
        torch.autograd.backward([s, y], [ds, dy])
        torch.autograd.backward([s64, y64], [ds.double(), dy.double()])
    else:
        y.backward(dy)
        y64.backward(dy.double())
    assert torch.equal(s.detach().double(), s64.detach())
    assert _err(y, y64) < 3e-3
    for a, g in zip(ins, ref):
        assert _err(a.grad, g.grad) < 3e-3
