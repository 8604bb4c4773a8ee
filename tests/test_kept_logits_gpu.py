"""What losses hold between forward and backward: the bound on kept logits is one for all that are alive."""
import gc

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_many_losses_before_one_backward(monkeypatch):
    from flextrain_b200.ops import cuda_ops
    n, h, v = 1024, 64, 8192
    logits = n * v * 2
    monkeypatch.setattr(cuda_ops._LinearCrossEntropy, "KEEP_BYTES", 2 * logits)
    gen = torch.Generator("cuda").manual_seed(0)
    w = (0.1 * torch.randn(v, h, generator=gen, device="cuda")).bfloat16().requires_grad_()
    labels = torch.randint(0, v, (n,), generator=gen, device="cuda")
    xs = [torch.randn(n, h, generator=gen, device="cuda").bfloat16().requires_grad_() for _ in range(6)]

    gc.collect()                                         # what other tests left would count as freed here

    def held():
        before = torch.cuda.memory_allocated()
        out = [cuda_ops.linear_cross_entropy(x, w, labels) for x in xs]
        return out, (torch.cuda.memory_allocated() - before) / logits

    want = [torch.autograd.grad(cuda_ops.linear_cross_entropy(x, w, labels), (x, w)) for x in xs]
    for _ in range(2):                                   # given back by a backward ...
        losses, kept = held()
        assert 2 <= kept < 2.5
        for i in (3, 0, 5, 1, 4, 2):
            for a, b in zip(torch.autograd.grad(losses[i], (xs[i], w)), want[i]):
                assert torch.equal(a, b)
    losses, kept = held()                                # ... while the losses themselves are still there
    assert 2 <= kept < 2.5
    del losses                                           # or by being dropped
    losses, kept = held()
    assert 2 <= kept < 2.5
    with torch.no_grad():
        del losses
        assert held()[1] < 0.5
    losses, kept = held()
    assert 2 <= kept < 2.5
