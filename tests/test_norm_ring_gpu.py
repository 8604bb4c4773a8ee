"""The norm backward's shared-memory ring: fewer steps than stages, several rounds of the ring, a last
step that is not full, each launch shape (1, 2 and 4 pieces per thread), with and without the
residual gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,rows", [(8, 1), (256, 5), (776, 2371), (1600, 148 * 4 * 6 + 3), (5120, 148 * 4 * 5 + 1),
                                    (5128, 299), (8192, 148 * 2 * 7 + 1), (8200, 150), (16384, 148 * 8 + 1)])
@pytest.mark.parametrize("ln", [False, True])
@pytest.mark.parametrize("residual", [False, True])
def test_norm_backward_ring(h, rows, ln, residual):
    from flextrain_b200.ops import cuda_ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(h + rows)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()     # noqa: E731
    x, w, dy, ds = rand(rows, h).requires_grad_(), (1 + 0.1 * rand(h)).detach().requires_grad_(), rand(rows, h), rand(rows, h)
    b = rand(h).requires_grad_() if ln else None
    x64, w64, b64 = (t.detach().double().requires_grad_() if t is not None else None for t in (x, w, b))
    if ln:
        y64 = torch.nn.functional.layer_norm(x64, (h,), w64, b64, 1e-5)
    else:
        y64 = x64 * torch.rsqrt(x64.pow(2).mean(-1, keepdim=True) + 1e-5) * w64
    if residual:
        s, y = cuda_ops.add_layernorm(x, torch.zeros_like(x), w, b, 1e-5) if ln else \
            cuda_ops.add_rmsnorm(x, torch.zeros_like(x), w, 1e-5)
        torch.autograd.backward([s, y], [ds, dy])
        torch.autograd.backward([x64 * 1, y64], [ds.double(), dy.double()])
    else:
        y = cuda_ops.layernorm(x, w, b, 1e-5) if ln else cuda_ops.rmsnorm_rows(x, w, 1e-5)
        y.backward(dy)
        y64.backward(dy.double())
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    for got, want in ((x, x64), (w, w64), (b, b64)):
        if got is not None:
            # one bf16 rounding of an fp32 expression: 2^-9 an element at most
            assert (got.grad.double() - want.grad).norm() <= 2.2e-3 * want.grad.norm() + 1e-3
