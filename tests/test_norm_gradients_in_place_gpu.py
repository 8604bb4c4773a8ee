"""Norm backward with its three ways out: parameter gradients added to what .grad holds, dx in two buffers for two
leaves, and the residual branch's gradient added inside (``norm_residual``), against fp32 PyTorch.

Tolerances: a 16-bit result is one rounding of an fp32 sum, 2^-9 relative to the largest term for bf16 (2^-12 fp16);
0.01 leaves room for the norm's own stored statistics, as in ``test_gpt_gpu.py``."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def _norm(x, w, b):
    if b is None:
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, 1e-5)


# one row, a ragged last step, eight narrow rows a step, the widest of each launch shape
@pytest.mark.parametrize("rows,h", [(1, 256), (37, 1600), (3001, 1600), (150, 5120), (9, 8192), (5, 16384)])
@pytest.mark.parametrize("ln", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_backward_into_existing_gradients(rows, h, ln, dtype):
    from flextrain_b200.ops import cuda_ops as ops
    g = torch.Generator(device="cuda").manual_seed(rows + h)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)                  # noqa: E731
    x, r, ds, dy, w0, b0 = rand(rows, h), rand(rows, h), rand(rows, h), rand(rows, h), rand(h), rand(h)
    held = rand(h), rand(h)

    def run(op, oracle, leaves):
        w, b = w0.clone().requires_grad_(), b0.clone().requires_grad_() if ln else None
        w.grad = gw = held[0].clone()
        if ln:
            b.grad = held[1].clone()
        mine = [t.clone().requires_grad_() for t in leaves]
        torch.autograd.backward(op(*mine, w, b), (ds, dy))
        wf, bf = w0.double().requires_grad_(), b0.double().requires_grad_() if ln else None
        ref = [t.double().requires_grad_() for t in leaves]
        torch.autograd.backward(oracle(*ref, wf, bf), (ds.double(), dy.double()))
        for a, b_ in zip(mine, ref):
            assert _rel(a.grad, b_.grad) < 0.01
        assert w.grad is gw and _rel(w.grad, held[0].double() + wf.grad) < 0.01
        if ln:
            assert _rel(b.grad, held[1].double() + bf.grad) < 0.01
        assert len({t.grad.data_ptr() for t in mine}) == len(mine)

    run(lambda x, w, b: ops.norm_residual(x, w, b, 1e-5), lambda x, w, b: (x * 1, _norm(x, w, b)), [x])
    # the kernel norms the rounded sum; its oracle likewise
    s = (x.float() + r.float()).to(dtype).double()
    run(lambda x, r, w, b: (ops.add_layernorm(x, r, w, b, 1e-5) if ln else ops.add_rmsnorm(x, r, w, 1e-5)),
        lambda x, r, w, b: (lambda t: (t, _norm(t, w, b)))(x + r + (s - (x + r)).detach()), [x, r])
