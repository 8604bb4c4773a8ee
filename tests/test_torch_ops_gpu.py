"""What the C++ autograd nodes owe PyTorch: saved-tensor hooks, the version check of in-place ops,
partial and repeated backward passes, strided inputs, refused transforms and types."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _r(*s, grad=True):
    return torch.randn(*s, device="cuda").bfloat16().requires_grad_(grad)


def _block(x, p):
    from flextrain_b200.ops import functional as F
    h = F.layernorm(x, p["w"], p["b"], 1e-5)
    qkv = F.bias_add(F.linear(h, p["wqkv"]), p["bqkv"])
    a = F.attention_packed(qkv, 2, 2, 64)
    s, h = F.add_rmsnorm(x, F.linear(a, p["wo"]), p["w"], 1e-5)
    return F.linear_add(F.swiglu(F.linear(h, p["wgu"])), p["wd"], s)


def _params():
    h, f = 128, 192
    return dict(w=_r(h), b=_r(h), wqkv=_r(3 * h, h), bqkv=_r(3 * h), wo=_r(h, h), wgu=_r(2 * f, h), wd=_r(h, f))


def test_saved_tensor_hooks_see_everything_and_change_nothing():
    x, p, dy = _r(2, 33, 128), _params(), _r(2, 33, 128, grad=False)
    ins = [x, *p.values()]
    want = torch.autograd.grad(_block(x, p), ins, dy)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(1) or t.cpu(), lambda t: t.cuda()):
        y = _block(x, p)
    got = torch.autograd.grad(y, ins, dy)
    assert len(seen) > 15
    for a, b in zip(got, want):
        assert (a.float() - b.float()).norm() <= 1e-3 * b.float().norm()      # dQ is summed in another order
    y = torch.utils.checkpoint.checkpoint(_block, x, p, use_reentrant=False)
    for a, b in zip(torch.autograd.grad(y, ins, dy), want):
        assert (a.float() - b.float()).norm() <= 1e-3 * b.float().norm()


def test_in_place_ops_follow_the_version_rules():
    from flextrain_b200.ops import functional as F
    leaf, bias = _r(4, 64), _r(64)
    with pytest.raises(RuntimeError, match="leaf"):
        F.bias_add(leaf, bias)
    x = leaf * 1
    y = x * x                                             # saves x
    out = F.bias_add(x, bias)
    assert out.data_ptr() == x.data_ptr()
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        (y.sum() + out.sum()).backward()
    with torch.no_grad():
        t = torch.zeros(4, 64, device="cuda").bfloat16()
        assert F.bias_add(t, bias).data_ptr() == t.data_ptr() and torch.equal(t[1], bias)


@pytest.mark.parametrize("frozen", ["x", "w", "res"])
def test_frozen_inputs_get_no_gradient(frozen):
    from flextrain_b200.ops import functional as F
    t = dict(x=_r(70, 64), w=_r(48, 64), res=_r(70, 48))
    t[frozen].requires_grad_(False)
    F.linear_add(t["x"], t["w"], t["res"]).backward(_r(70, 48, grad=False))
    for n, v in t.items():
        assert (v.grad is None) == (n == frozen)


def test_an_existing_gradient_buffer_is_accumulated_into():
    from flextrain_b200.ops import functional as F
    x, w = _r(40, 64, grad=False), _r(64, 64)
    dy = _r(40, 64, grad=False)
    F.linear(x, w).backward(dy)
    first = w.grad.clone()
    buf = w.grad
    F.linear(x, w).backward(dy)
    assert w.grad is buf
    assert (buf.float() - 2 * first.float()).norm() <= 5e-3 * buf.float().norm()


def test_strided_inputs():
    from flextrain_b200.ops import functional as F
    w, wide = _r(48, 64), _r(30, 200, grad=False)
    dy = _r(48, 30, grad=False).t()
    for x in (wide[:, :64], wide[:, 8:72], _r(64, 30, grad=False).t()):
        y = F.linear(x, w)
        assert (y.float() - x.float() @ w.float().t()).norm() <= 5e-3 * y.float().norm()
        (g,) = torch.autograd.grad(y, w, dy)
        want = dy.float().t() @ x.float()
        assert (g.float() - want).norm() <= 5e-3 * want.norm()


def test_refusals_stay_refusals():
    from flextrain_b200.ops import functional as F
    with pytest.raises(TypeError):
        F.linear(torch.randn(4, 64, device="cuda"), torch.randn(8, 64, device="cuda"))
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.vmap(lambda t: F.linear(t, _r(8, 64, grad=False)))(_r(2, 4, 64, grad=False))
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.jvp(lambda t: F.swiglu(t), (_r(4, 64, grad=False),), (_r(4, 64, grad=False),))
    with pytest.raises(RuntimeError):
        F.layernorm(_r(4, 20), _r(20), _r(20), 1e-5)     # a width that is no multiple of 8
