"""The backward's split of a kv head's query heads over CTAs: the rule (restated here and compared
with the library's) and the gradients at shapes with one part, equal parts and a smaller last part."""
import pytest
import torch


def splits(b, s, hq, hkv):
    """csrc/kernels/attention.cu, ft_attn_bwd_splits."""
    blocks, heads = -(-s // 128), hq // hkv
    n = min(-(-296 // (b * hkv * (blocks + 1))), heads)
    return -(-heads // -(-heads // n))


@pytest.mark.parametrize("b", [1, 3])
@pytest.mark.parametrize("s", [1, 128, 1000, 4096, 32768])
@pytest.mark.parametrize("hq,hkv", [(1, 1), (32, 32), (64, 8), (45, 1), (7, 1), (48, 4)])
def test_every_part_has_heads_and_jobs_are_even(b, s, hq, hkv):
    n, heads, blocks = splits(b, s, hq, hkv), hq // hkv, -(-s // 128)
    part = -(-heads // n)
    assert 1 <= n <= heads and (n - 1) * part < heads <= n * part
    share = heads * b * hkv * blocks * (blocks + 1) / 2 / 148
    assert part == 1 or (part - 1) * blocks <= 2 * share   # no part is much longer than an SM's share
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    assert not cuda_lib_available() or cuda_lib().ft_attn_bwd_splits(b, s, hq, hkv) == n
    # scratch: bounded by what it is for
    assert 2 * n * b * s * hkv * 128 * 4 <= 2 * 128 * 4 * 128 * (296 + 2 * b * hkv * blocks)


def parts_of(b, s, hq, hkv, d):
    """csrc/kernels/attention.cu, ft_attn_bwd_parts."""
    blocks, heads, groups = -(-s // 128), hq // hkv, b * hkv
    total, fixed, times = groups * heads * blocks * (blocks + 1) / 2, 5, {}
    for n in range(1, splits(b, s, hq, hkv) + 1):
        part, jobs = -(-heads // n), groups * n * blocks
        if (n - 1) * part < heads:
            t = part * blocks + fixed
            t = max(t, (total + jobs * fixed) / 148 + fixed / 2) if jobs > 148 else t
            times[n] = t + (n > 1) * (1.5 + (1.5 if d == 128 else 1.0) * jobs / 148)
    return min(times, key=times.get)


# (b, s, hq, hkv, d): the division that measured best.  The first six were slower divided.
@pytest.mark.parametrize("shape,best", [((1, 256, 160, 40, 64), 1), ((1, 512, 320, 40, 64), 1), ((10, 512, 8, 4, 128), 1), ((8, 1024, 8, 4, 64), 1), ((3, 1000, 16, 8, 128), 1),
                                        ((1, 128, 16, 8, 128), 1), ((1, 4096, 16, 8, 128), 1), ((1, 2048, 8, 1, 64), 8),
                                        ((1, 2048, 64, 8, 128), 2), ((2, 4096, 64, 8, 128), 1), ((1, 1024, 32, 32, 64), 1)])
def test_heads_are_divided_where_it_is_faster(shape, best):
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    assert parts_of(*shape) == best
    if cuda_lib_available():
        for b in (1, 2, 3, 8):
            for s in (1, 128, 300, 1000, 2048, 4096):
                for hq, hkv in ((8, 1), (45, 1), (7, 1), (32, 8), (64, 8), (16, 8), (12, 12), (28, 4)):
                    for d in (64, 128):
                        assert cuda_lib().ft_attn_bwd_parts(b, s, hq, hkv, d) == parts_of(b, s, hq, hkv, d)


@pytest.mark.gpu
@pytest.mark.parametrize("b,s,hq,hkv,d,parts", [(1, 300, 5, 1, 64, 5), (1, 1000, 45, 1, 128, 23), (2, 1300, 28, 4, 64, 4),
                                                (1, 2048, 64, 8, 128, 3), (2, 4096, 8, 8, 64, 1)])
@pytest.mark.parametrize("packed", [False, True])
def test_gradients(b, s, hq, hkv, d, parts, packed):
    from flextrain_b200.ops import functional as F
    from flextrain_b200.ops.native import cuda_lib
    assert splits(b, s, hq, hkv) == parts == cuda_lib().ft_attn_bwd_splits(b, s, hq, hkv)
    gen = torch.Generator(device="cuda").manual_seed(s)
    qkv = torch.randn(b, s, (hq + 2 * hkv) * d, generator=gen, device="cuda").bfloat16().requires_grad_()
    dy = torch.randn(b, s, hq * d, generator=gen, device="cuda").bfloat16()
    q, k, v = (t.unflatten(-1, (-1, d)) for t in qkv.split([hq * d, hkv * d, hkv * d], -1))
    out = F.attention_packed(qkv, hq, hkv, d) if packed else F.causal_attention(q, k, v).flatten(2)
    (got,) = torch.autograd.grad(out, qkv, dy)
    ref = qkv.detach().double().requires_grad_()
    q, k, v = (t.unflatten(-1, (-1, d)).transpose(1, 2) for t in ref.split([hq * d, hkv * d, hkv * d], -1))
    mask = torch.ones(s, s, dtype=torch.bool, device="cuda").triu(1)
    want = torch.zeros_like(ref)
    for i in range(b):                                    # one kv head at a time
        for j in range(hkv):
            r = slice(j * hq // hkv, (j + 1) * hq // hkv)
            sc = (q[i, r] @ k[i, j].T / d ** 0.5).masked_fill(mask, float("-inf")).softmax(-1)
            o = (sc @ v[i, j]).transpose(0, 1).flatten(1)
            (g,) = torch.autograd.grad(o, ref, dy[i, :, r.start * d:r.stop * d].double(), retain_graph=True)
            want += g
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    for a, c in zip(got.split([hq * d, hkv * d, hkv * d], -1), want.split([hq * d, hkv * d, hkv * d], -1)):
        # four times what bf16 probabilities and gradients leave (0.0025)
        assert (a.double() - c).norm() <= 0.01 * c.norm()
