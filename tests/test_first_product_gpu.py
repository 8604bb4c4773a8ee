"""Blocks whose first weight is still being gathered (``_ft_gather``, set by the parameter coordinator on
several GPUs), with an ordinary product in place of the all-gather GEMM: outputs and gradients are those
of the same block with a complete weight, with gradients recorded directly and through the engine's
recompute."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Pending:
    """As memory/coordinator/parameter.py's _PendingFirstGemm, on a weight that is complete already."""

    def __init__(self, w, covered):
        self.w, self.covered, self.calls = w, covered, []

    def covers(self, rows, cols):
        return self.covered

    def run(self, x2, out):
        from flextrain_b200.ops.cuda_ops import gemm
        self.calls.append("run")
        self.w._ft_gather = None
        gemm(x2, False, self.w, False, x2.shape[0], self.w.shape[0], x2.shape[1], out=out)

    def complete_without_product(self):
        self.calls.append("complete")
        self.w._ft_gather = None


def _block(kind):
    from flextrain_b200.models import gpt, llama
    from flextrain_b200.ops import functional as F
    torch.manual_seed(3)
    if kind == "gpt":
        mod = gpt.GPTBlock(gpt.GPTConfig(num_layers=1, hidden=256, num_heads=4, ffn=512, vocab=64, seq_len=160),
                           dtype=torch.bfloat16)
        return mod.cuda(), ()
    mod = llama.LlamaBlock(llama.LlamaConfig(num_layers=1, hidden=256, num_heads=4, num_kv_heads=2, ffn=512, vocab=64,
                                             seq_len=160), dtype=torch.bfloat16)
    return mod.cuda(), F.rope_tables(160, 64, 10000.0, device=torch.device("cuda"))


@pytest.mark.parametrize("kind", ["gpt", "llama"])
@pytest.mark.parametrize("covered", [True, False])
@pytest.mark.parametrize("recompute", [False, True])
def test_block(kind, covered, recompute):
    from flextrain_b200.checkpointing import checkpointed_backward, checkpointed_forward
    mod, extra = _block(kind)
    with torch.no_grad():
        for p in mod.parameters():
            p.normal_(0.0 if p.dim() > 1 else 0.5, 0.1)
    x, dy = (torch.randn(2, 160, 256, device="cuda").bfloat16() for _ in range(2))
    got = {}
    for pending in (False, True):
        gather = _Pending(mod.wqkv, covered) if pending else None
        mod.zero_grad(set_to_none=True)
        leaf = x.clone().requires_grad_()
        mod.wqkv._ft_gather = gather
        if recompute:
            y, ctx = checkpointed_forward(mod, leaf, *extra)
            if pending:
                assert gather.calls == ["run" if covered else "complete"]
            mod.wqkv._ft_gather = gather
            dx = checkpointed_backward(ctx, dy)[0]
        else:
            y = mod(leaf, *extra)
            y.backward(dy)
            dx = leaf.grad
        if pending:
            assert gather.calls == ["run" if covered else "complete"] * (2 if recompute else 1)
        got[pending] = [y.detach(), dx, *(p.grad for p in mod.parameters())]
    torch.cuda.synchronize()
    for a, b in zip(got[True], got[False]):
        # the GPT block rounds once more between product and bias (2^-9 per element), and dQ is summed in
        # another order: a change of single roundings that travels through two more products
        assert (a.double() - b.double()).norm() <= 1e-2 * b.double().norm()
