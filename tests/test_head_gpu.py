"""Head and loss: the row kernels at their edges, the kept logits of the last chunk, a second backward."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v", [8, 1000, 1003, 4104, 16392])     # below, at and past four pieces per thread; a tail
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_row_kernels(v, dtype):
    from flextrain_b200.ops.native import cuda_lib, dtype_code, ptr, stream_handle
    rows, ld, lib = 37, (v + 7) // 8 * 8, cuda_lib()
    gen = torch.Generator(device="cuda").manual_seed(v)
    logits = (3 * torch.randn(rows, ld, generator=gen, device="cuda")).to(dtype)
    logits[0, : v // 2] = float("-inf")                  # a masked half
    logits[1, :] = torch.finfo(dtype).min                # masked with the type's lowest value
    logits[2, v // 3] = float("nan")
    logits[3, v - 1] = float("inf")
    logits[4, :] = float("-inf")
    labels = torch.randint(0, v, (rows,), generator=gen, device="cuda")
    labels[0], labels[5], labels[6] = v - 1, -100, v     # ignored, and out of range: ignored too
    x = logits[:, :v].double()
    lse, total = torch.empty(rows, device="cuda"), torch.zeros(1, device="cuda")
    assert lib.ft_xent_fwd(ptr(logits), ld, ptr(labels), rows, v, -100, ptr(lse), ptr(total), dtype_code(dtype),
                           stream_handle()) == 0
    want = x.logsumexp(1)
    ok = torch.ones(rows, dtype=torch.bool, device="cuda")
    ok[2:5] = False                                      # NaN, +inf and nothing but -inf: no softmax
    assert lse[~ok].isnan().all()
    assert torch.allclose(lse[ok].double(), want[ok], rtol=1e-6, atol=1e-5)
    keep = logits.clone()
    scale = torch.full((1,), 0.5, device="cuda")
    lse = want.float()
    assert lib.ft_xent_bwd(ptr(logits), ld, ptr(labels), rows, v, -100, ptr(lse), ptr(scale), 1.0, dtype_code(dtype),
                           stream_handle()) == 0
    valid = (labels >= 0) & (labels < v)
    hot = torch.zeros(rows, v, dtype=torch.float64, device="cuda")
    hot[valid] = torch.nn.functional.one_hot(labels[valid], v).double()
    grad = (x - want[:, None]).exp().sub(hot) * 0.5 * valid[:, None]
    # one rounding to the type, and e^x of an argument that fp32 holds to 2^-20
    tol = 2.0 ** (-8 if dtype == torch.bfloat16 else -11) * 1.1
    sel = ok & (torch.arange(rows, device="cuda") != 1)
    assert ((logits[sel, :v].double() - grad[sel]).abs() <= tol * grad[sel].abs() + 1e-7).all()
    assert torch.equal(logits[:, v:], keep[:, v:])


@pytest.mark.parametrize("n", [1, 129, 4096, 4097, 8192])       # one chunk, a part of one, one and a row, two whole
def test_kept_logits_change_nothing(n, monkeypatch):
    from flextrain_b200.ops import cuda_ops
    h, v = 64, 1024
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, h, generator=gen, device="cuda").bfloat16().requires_grad_()
    w = (0.1 * torch.randn(v, h, generator=gen, device="cuda")).bfloat16().requires_grad_()
    labels = torch.randint(0, v, (n,), generator=gen, device="cuda")

    def grads(twice=False):
        loss = cuda_ops.linear_cross_entropy(x, w, labels)
        res = [torch.autograd.grad(loss, (x, w), retain_graph=twice)]
        if twice:                                        # the kept buffer holds gradients by now
            res.append(torch.autograd.grad(loss, (x, w)))
        return res

    first, second = grads(twice=True)
    monkeypatch.setattr(cuda_ops._LinearCrossEntropy, "KEEP_BYTES", 0)
    (plain,) = grads()
    for a, b, c in zip(first, second, plain):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("rows", [37, 4100])                    # one chunk, whose logits are kept, and two
def test_a_backward_pass_for_chosen_inputs_changes_no_other(rows):
    from flextrain_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 64, generator=gen, device="cuda").bfloat16().requires_grad_()
    w = (0.1 * torch.randn(104, 64, generator=gen, device="cuda")).bfloat16().requires_grad_()
    labels = torch.randint(0, 104, (rows,), generator=gen, device="cuda")
    F.linear_cross_entropy(x, w, labels).backward()
    dx, dw = x.grad, w.grad
    w.grad = held = torch.ones_like(w)
    assert torch.equal(torch.autograd.grad(F.linear_cross_entropy(x, w, labels), x)[0], dx) and (held == 1).all()
    for got, want in zip(torch.autograd.grad(F.linear_cross_entropy(x, w, labels), (x, w)), (dx, dw)):
        assert torch.equal(got, want)
    assert (held == 1).all()
    x.grad = None
    F.linear_cross_entropy(x, w, labels).backward(inputs=[x])
    assert torch.equal(x.grad, dx) and (held == 1).all()
    F.linear_cross_entropy(x, w, labels).backward(inputs=[w])
    assert w.grad is held and torch.equal(x.grad, dx)
    assert (held.double() - 1 - dw.double()).abs().max() <= 2 ** -7      # one rounding of a value near 1
