"""Attention over tensors whose batches or tokens do not follow one another in memory, forward and
backward, against the same values in a contiguous tensor."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _r(*s):
    return torch.randn(*s, generator=torch.Generator("cuda").manual_seed(sum(s)), device="cuda").bfloat16()


LAYOUTS = {
    "prefix": lambda b, s, w: _r(b, s + 3, w)[:, :s],
    "tokens first": lambda b, s, w: _r(s, b, w).transpose(0, 1),
    "columns": lambda b, s, w: _r(b, s, 2 * w)[..., w:],
    "one sequence": lambda b, s, w: _r(1, s, w).expand(b, s, w),
}


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("b,s", [(2, 200), (1, 129), (3, 1)])
@pytest.mark.parametrize("packed", [True, False])
def test_gradients(layout, b, s, packed):
    from flextrain_b200.ops import functional as F
    from flextrain_b200.ops.native import cuda_lib
    t, dy = LAYOUTS[layout](b, s, 6 * 64), _r(b, s, 4 * 64)
    got = []
    for x in (t.detach(), t.contiguous()):
        x.requires_grad_()
        if packed:
            y = F.attention_packed(x, 4, 1, 64)
            g = torch.autograd.grad(y, x, dy)
        else:
            parts = [p.unflatten(-1, (-1, 64)) for p in x.split([256, 64, 64], -1)]
            y = F.causal_attention(*parts).flatten(2)
            g = torch.autograd.grad(y, parts, dy)
        got.append((y, *g))
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    assert torch.equal(got[0][0], got[1][0])
    for a, c in zip(got[0][1:], got[1][1:]):          # dQ is summed in another order
        assert (a.float() - c.float()).norm() <= 2e-3 * c.float().norm()
