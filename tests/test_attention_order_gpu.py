"""The CTA order of the causal attention grids (chunks of heads, heaviest blocks first): every (head,
block) job runs exactly once.  On the CPU as arithmetic, on the GPU where a grid has several chunks."""
import pytest
import torch


def _job(idx, heads, blocks, chunk):
    """csrc/kernels/attention_common.cuh, causal_job."""
    c = idx // (chunk * blocks)
    first = c * chunk
    n = min(chunk, heads - first)
    r = idx - c * chunk * blocks
    return first + r % n, r // n


def _chunk(heads, size):
    """csrc/kernels/attention_common.cuh, causal_chunk."""
    c = min(max((64 << 20) // max(size, 1), 16), heads)
    return -(-heads // -(-heads // c))


@pytest.mark.parametrize("heads", [1, 2, 15, 16, 17, 33, 160, 323])
@pytest.mark.parametrize("blocks", [1, 3, 16])
@pytest.mark.parametrize("size", [1, 1 << 20, 3 << 20, 64 << 20, 1 << 33])
def test_every_job_once_and_heavy_first(heads, blocks, size):
    chunk = _chunk(heads, size)
    assert 1 <= chunk <= heads
    jobs = [_job(i, heads, blocks, chunk) for i in range(heads * blocks)]
    assert sorted(jobs) == [(h, r) for h in range(heads) for r in range(blocks)]
    for a, b in zip(jobs, jobs[1:]):
        assert b[1] >= a[1] or b[0] // chunk > a[0] // chunk


@pytest.mark.gpu
@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 129, 1, 1, 64), (3, 300, 7, 7, 128), (2, 4224, 20, 20, 128)])
def test_attention_over_several_chunks(b, s, hq, hkv, d):
    """The last shape: 40 heads of 2.2 MB of keys and values, in two chunks of the forward and three
    of the backward; against fp64, at four times the distance bf16 rounding leaves (0.0025)."""
    from flextrain_b200.ops.functional import causal_attention
    gen = torch.Generator(device="cuda").manual_seed(s)
    q, k, v, dy = (torch.randn(b, s, h, d, generator=gen, device="cuda").bfloat16() for h in (hq, hkv, hkv, hq))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    out = causal_attention(*leaves)
    out.backward(dy)
    ref = [t.detach().double().requires_grad_() for t in leaves]
    rep = hq // hkv
    mask = torch.ones(s, s, dtype=torch.bool, device="cuda").triu(1)
    for i in range(b):
        for h in range(hq):
            sc = (ref[0][i, :, h] @ ref[1][i, :, h // rep].T) / d ** 0.5
            o = sc.masked_fill(mask, float("-inf")).softmax(-1) @ ref[2][i, :, h // rep]
            o.backward(dy[i, :, h].double())
            assert (out[i, :, h].double() - o).norm() < 0.01 * o.norm()
    for got, want in zip(leaves, ref):
        assert (got.grad.double() - want.grad).norm() < 0.01 * want.grad.norm()
