"""A GPT block as one autograd node against the same block op by op: the kernels and their order are the same, so every
value is, except where the attention backward adds dq up in the order in which its CTAs arrive (sequences of more than one
block of 128)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NAMES = ("x", "ln1_w", "ln1_b", "wqkv", "bqkv", "wo", "bo", "ln2_w", "ln2_b", "w_fc", "b_fc", "w_proj", "b_proj")


def _block(hidden=256, heads=4, ffn=1024, dtype=torch.bfloat16, held=True, seed=0):
    from flextrain_b200.models.gpt import GPTBlock, GPTConfig
    gen = torch.Generator(device="cuda").manual_seed(seed)
    with torch.device("cuda"):
        m = GPTBlock(GPTConfig(num_layers=1, hidden=hidden, num_heads=heads, ffn=ffn, vocab=64, seq_len=64), dtype=dtype)
    for p in m.parameters():
        p.data.normal_(1.0 if p.dim() == 1 else 0.0, 0.05, generator=gen)
        if held:
            p.grad = torch.empty_like(p).normal_(0, 1, generator=gen)
    return m


def _pass(m, x, dy, one, monkeypatch, run=None):
    from flextrain_b200.ops import functional as F
    taken = []
    real = F.gpt_block
    monkeypatch.setattr(F, "gpt_block", lambda *a: (taken.append(real(*a)), taken[-1])[1] if one else None)
    y = m(x)
    assert not one or taken[-1] is not None
    (run or (lambda t: t.backward(dy)))(y)
    torch.cuda.synchronize()
    from flextrain_b200.ops.native import cuda_lib
    assert cuda_lib().ft_gemm_error() == 0
    monkeypatch.setattr(F, "gpt_block", real)
    return [y.detach(), x.grad] + [p.grad for p in m.parameters()]


def _both(monkeypatch, shape, exact=True, run=None, leaf=True, tie=(), **kw):
    out = []
    for one in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(5)
        m = _block(**kw)
        for a, b in tie:
            setattr(m, b, getattr(m, a))
        x = torch.randn(*shape, generator=gen, device="cuda").to(kw.get("dtype", torch.bfloat16)).requires_grad_(leaf)
        dy = torch.randn(*shape, generator=gen, device="cuda").to(x.dtype)
        out.append(_pass(m, x, dy, one, monkeypatch, run and (lambda y, m=m, x=x, dy=dy: run(y, m, x, dy))))
    for a, b in zip(*out):
        assert (a is None) == (b is None)
        if a is not None:
            # dq sums in another order: a rounding of the 16-bit type here and there, and what follows from it
            assert torch.equal(a, b) if exact else (a - b).float().norm() <= 2e-3 * a.float().norm()


@pytest.mark.parametrize("shape,kw", [((2, 128, 256), {}), ((1, 1, 128), dict(hidden=128, heads=2, ffn=72)), ((3, 77, 256), dict(heads=2)),
                                      ((2, 100, 768), dict(hidden=768, heads=12, ffn=3072)), ((1, 65, 256), dict(ffn=128))])
@pytest.mark.parametrize("held", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_the_same_values(monkeypatch, shape, kw, held, dtype):
    _both(monkeypatch, shape, held=held, dtype=dtype, **kw)


def test_long_sequences(monkeypatch):
    _both(monkeypatch, (2, 300, 256), exact=False)


def test_an_input_without_gradient(monkeypatch):
    _both(monkeypatch, (2, 64, 256), leaf=False)


@pytest.mark.parametrize("tie", [[("ln1_w", "ln2_w")], [("ln1_b", "ln2_b")], [("ln1_w", "ln2_w"), ("ln1_b", "ln2_b")],
                                 [("ln1_w", "ln2_b")]])
@pytest.mark.parametrize("held", [True, False])
def test_one_parameter_in_both_norms(monkeypatch, tie, held):
    _both(monkeypatch, (2, 100, 768), tie=tie, held=held, hidden=768, heads=12, ffn=3072)


def test_backward_twice_and_chosen_gradients(monkeypatch):
    _both(monkeypatch, (2, 64, 256), run=lambda y, m, x, dy: (y.backward(dy, retain_graph=True), y.backward(dy)))

    def chosen(y, m, x, dy):
        before = [p.grad.clone() for p in m.parameters()]
        got = torch.autograd.grad(y, [x, m.ln1_b, m.b_fc], dy)
        x.grad = torch.cat([g.flatten() for g in got])[:x.numel()].view_as(x)
        assert all(torch.equal(p.grad, b) for p, b in zip(m.parameters(), before))
    _both(monkeypatch, (2, 64, 256), run=chosen)


@pytest.mark.parametrize("names", [(n,) for n in NAMES] + [("x", "wo"), ("w_fc", "b_proj")])
def test_a_backward_pass_for_chosen_inputs(monkeypatch, names):
    def run(y, m, x, dy):
        before = {n: p.grad.clone() for n, p in m.named_parameters()}
        y.backward(dy, inputs=[x if n == "x" else getattr(m, n) for n in names])
        changed = {n for n, p in m.named_parameters() if not torch.equal(p.grad, before[n])} | ({"x"} if x.grad is not None else set())
        assert changed == set(names)
    _both(monkeypatch, (2, 100, 256), run=run)


def test_hooks_see_what_they_saw(monkeypatch):
    def run(y, m, x, dy):
        seen = []
        m.ln2_w.register_hook(lambda g: seen.append(g.clone()) or g * 2)
        m.b_proj.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad.clone()))
        y.backward(dy)
        assert len(seen) == 2
    _both(monkeypatch, (2, 64, 256), run=run)


def test_saved_tensors_go_through_their_hooks(monkeypatch):
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t), t.cpu())[1], lambda t: t.cuda()):
        _both(monkeypatch, (2, 64, 256), held=False)
    assert len(packed) > 12


def test_blocks_that_stay_op_by_op():
    from flextrain_b200.ops import functional as F
    m = _block()
    args = list(m.parameters())
    x = torch.randn(1, 64, 256, device="cuda").bfloat16().requires_grad_()
    assert F.gpt_block(x, args, 4, 1e-5) is not None
    with torch.no_grad():
        assert F.gpt_block(x, args, 4, 1e-5) is None
    assert F.gpt_block(x, args, 8, 1e-5) is None               # heads of 32
    assert F.gpt_block(x.float(), args, 4, 1e-5) is None
    m.bo.requires_grad_(False)
    assert F.gpt_block(x, args, 4, 1e-5) is None
    m.bo.requires_grad_(True)
    m.wqkv._ft_gather = object()
    assert F.gpt_block(x, args, 4, 1e-5) is None
    big = torch.zeros(80000, 1, 256, device="cuda", dtype=torch.bfloat16)
    del m.wqkv._ft_gather
    assert F.gpt_block(big, args, 4, 1e-5) is None
