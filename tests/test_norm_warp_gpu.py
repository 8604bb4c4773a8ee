"""Norms of rows that a warp covers (up to 1024 values): each number of pieces a lane, rows that end inside a piece's lanes, fewer
rows than CTAs, than warps of a CTA, and several rows a warp; forward with one and with several rows a CTA; with and without
the residual gradient, and dx in two buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [8, 248, 256, 264, 512, 520, 768, 776, 1024])
@pytest.mark.parametrize("rows", [1, 147, 149, 1187, 1281, 4999])
@pytest.mark.parametrize("ln", [False, True])
@pytest.mark.parametrize("form", ["plain", "two leaves"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_norms(h, rows, ln, form, dtype):
    from flextrain_b200.ops import cuda_ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(h + rows)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)      # noqa: E731
    x, r, dy, ds = (rand(rows, h) for _ in range(4))
    w, b = (1 + 0.1 * rand(h)).requires_grad_(), rand(h).requires_grad_() if ln else None
    x.requires_grad_()
    r.requires_grad_()
    if form == "plain":
        s64 = x.detach().double().requires_grad_()
        y = cuda_ops.layernorm(x, w, b, 1e-5) if ln else cuda_ops.rmsnorm_rows(x, w, 1e-5)
        y.backward(dy)
    else:
        s, y = cuda_ops.add_layernorm(x, r, w, b, 1e-5) if ln else cuda_ops.add_rmsnorm(x, r, w, 1e-5)
        torch.autograd.backward([s, y], [ds, dy])
        assert torch.equal(s, x + r) and torch.equal(x.grad, r.grad) and x.grad.data_ptr() != r.grad.data_ptr()
        s64 = s.detach().double().requires_grad_()
    w64, b64 = (t.detach().double().requires_grad_() if t is not None else None for t in (w, b))
    y64 = torch.nn.functional.layer_norm(s64, (h,), w64, b64, 1e-5) if ln else \
        s64 * torch.rsqrt(s64.pow(2).mean(-1, keepdim=True) + 1e-5) * w64
    torch.autograd.backward([y64] if form == "plain" else [s64 * 1, y64], [dy.double()] if form == "plain" else [ds.double(), dy.double()])
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    # one rounding to 16 bits of an fp32 expression: half an ulp, 2^-8 of the value in bf16 and 2^-11 in fp16, an element at most
    # (just above a power of two), which a gradient of eight values comes near to
    tol = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    for got, want in ((y, y64), (x.grad, s64.grad), (w.grad, w64.grad), (b.grad if ln else None, b64.grad if ln else None)):
        if got is not None:
            assert (got.double() - want).norm() <= tol * want.norm() + 1e-3
