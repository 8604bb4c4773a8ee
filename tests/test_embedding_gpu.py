"""Embedding whose backward adds to a gradient that is there: repeated tokens, one token only (its columns divided over few and over many
CTAs, its rows over a CTA's threads), more rows than a CTA looks at at once, and what stays with the general way (no gradient yet, hooks, many tokens, chosen gradients)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(n, v, h, dtype, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    tokens = torch.randint(0, v, (1, n), generator=gen, device="cuda")
    ints = lambda *s: torch.randint(-3, 4, s, generator=gen, device="cuda").to(dtype)      # noqa: E731
    return tokens, ints(v, h).requires_grad_(), ints(1, n, h), ints(v, h)


@pytest.mark.parametrize("n,v,h", [(1, 1, 8), (300, 1, 768), (257, 7, 264), (1024, 50304, 768), (4096, 500, 2056), (513, 100, 8192),
                                   (4097, 300, 64), (100, 50, 8200),
                                   (4096, 1, 768), (4095, 3, 8), (1030, 2, 8192), (9, 1, 4104), (8, 1, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gradient(n, v, h, dtype):
    from flextrain_b200.ops import functional as F
    from flextrain_b200.ops.native import cuda_lib
    tokens, w, dy, held = _case(n, v, h, dtype)
    w.grad = held.clone()
    y = F.embedding(tokens, w)
    assert torch.equal(y, w.detach()[tokens])
    before, address = cuda_lib().ft_launch_count(), w.grad.data_ptr()
    y.backward(dy)
    torch.cuda.synchronize()
    assert (cuda_lib().ft_launch_count() - before == 1) == (n <= 4096 and h <= 8192)
    want = held.double().index_add_(0, tokens[0], dy[0].double())
    # sums of at most 4097 integers up to 3, exact in fp32; one rounding, or two where autograd adds
    one = want.to(dtype)
    assert torch.equal(w.grad, one) or not (n <= 4096 and h <= 8192)
    assert (w.grad.double() - want).abs().max() <= 2 ** (-7 if dtype == torch.bfloat16 else -10) * want.abs().max()
    assert w.grad.data_ptr() == address


def test_the_general_way_stays():
    from flextrain_b200.ops import functional as F
    tokens, w, dy, held = _case(64, 40, 64, torch.bfloat16)
    want = torch.zeros(40, 64, device="cuda", dtype=torch.float64).index_add_(0, tokens[0], dy[0].double())
    F.embedding(tokens, w).backward(dy)                           # no gradient yet
    assert torch.equal(w.grad, want.bfloat16())
    (g,) = torch.autograd.grad(F.embedding(tokens, w), w, dy)     # a chosen gradient is returned, .grad left alone
    assert torch.equal(g, want.bfloat16()) and torch.equal(w.grad, want.bfloat16())
    seen = []
    handle = w.register_hook(lambda t: seen.append(t))
    F.embedding(tokens, w).backward(dy)
    handle.remove()
    assert len(seen) == 1 and torch.equal(w.grad, (2 * want).bfloat16())
    with torch.no_grad():
        assert torch.equal(F.embedding(tokens, w), w[tokens])


def test_transforms_that_torch_has_stay():
    """Forward-mode derivatives, vmap and torch.func.grad of a table, with and without a gradient that is there."""
    import torch.autograd.forward_ad as fwd
    from flextrain_b200.ops import functional as F
    for has in (False, True):
        tokens, w, dy, held = _case(12, 40, 64, torch.bfloat16)
        w.grad = held.clone() if has else None
        t = held + 1
        y, dot = torch.func.jvp(lambda v: F.embedding(tokens, v), (w,), (t,))
        assert torch.equal(y, w[tokens]) and torch.equal(dot, t[tokens])
        with fwd.dual_level():
            dual = fwd.unpack_dual(F.embedding(tokens, fwd.make_dual(w, t)))
        assert torch.equal(dual.tangent, t[tokens])
        assert torch.equal(torch.func.vmap(lambda i: F.embedding(i, w))(tokens.view(3, 4)), w[tokens.view(3, 4)])
        got = torch.func.grad(lambda v: (F.embedding(tokens, v) * dy).sum())(w)
        assert torch.equal(got, torch.zeros_like(w).index_add_(0, tokens[0], dy[0]))
        assert w.grad is None if not has else torch.equal(w.grad, held)
