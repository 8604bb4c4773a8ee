"""Query tiles of a CTA in the forward attention of 64-wide heads: the rule (restated here with a queue of SMs and compared with the
library's), and both kernels at lengths that end inside a tile, with few jobs and with several for every SM."""
import heapq

import pytest
import torch


def tiles(heads, s):
    t = -(-s // 128)
    total = heads * t * (t + 1) / 2
    if t > 16 or total > 2000 * 148:
        return 2
    jobs = heads * t
    singles = 9000 + max(2700 * t, total / 148 * 2312) + (5000 * (jobs - 296) / 296 if jobs > 296 else 0)
    free, last = [0] * 148, t
    while last > 0:
        for _ in range(heads):
            heapq.heapreplace(free, free[0] + 3365 * last + 7000)
        last -= 1 if last % 2 else 2
    return 1 if singles < max(free) + 3000 else 2


def test_the_rule_is_the_librarys():
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    lib, seen = cuda_lib(), set()
    for heads in (1, 2, 7, 24, 48, 64, 75, 100, 147, 148, 149, 300, 777):
        for s in (1, 64, 128, 129, 300, 512, 1000, 1024, 1500, 2048):
            want = tiles(heads, s)
            assert lib.ft_attn_fwd_tiles(heads, s, 64) == want
            assert lib.ft_attn_fwd_tiles(heads, s, 128) == 2
            seen.add(want)
    assert seen == {1, 2}
    assert all(lib.ft_attn_fwd_tiles(h, s, 64) == 2 for h, s in ((4, 2049), (16, 4096), (1 << 20, 128)))


@pytest.mark.gpu
@pytest.mark.parametrize("b,s,h,kv", [(1, 1, 1, 1), (2, 127, 4, 4), (2, 128, 2, 1), (3, 129, 8, 2), (2, 512, 12, 12), (1, 1000, 25, 5),
                                      (3, 1000, 16, 16), (2, 300, 160, 160), (1, 2048, 4, 1), (1, 2100, 3, 3)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_forward_and_gradients(b, s, h, kv, dtype):
    from flextrain_b200.ops import functional as F
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(s + h)
    q, k, v, dy = (torch.randn(b, s, n, 64, generator=gen, device="cuda").to(dtype) for n in (h, kv, kv, h))
    ours = [t.requires_grad_() for t in (q, k, v)]
    y = F.causal_attention(*ours)
    y.backward(dy)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    ref = [t.detach().double().requires_grad_() for t in (q, k, v)]
    qh, kh, vh = (t.transpose(1, 2) for t in ref)
    kh, vh = (t.repeat_interleave(h // kv, 1) for t in (kh, vh))
    p = (qh @ kh.transpose(2, 3) / 8).masked_fill(torch.ones(s, s, dtype=torch.bool, device="cuda").triu(1), float("-inf")).softmax(-1)
    want = (p @ vh).transpose(1, 2)
    want.backward(dy.double())
    # P and the result are rounded to 16 bits (2^-9 or 2^-12 each on average), in the backward dS too
    tol = 0.006 if dtype == torch.bfloat16 else 0.001
    for got, ref_t in [(y, want)] + [(a.grad, r.grad) for a, r in zip(ours, ref)]:
        assert (got.double() - ref_t).norm() <= tol * ref_t.norm() + 1e-3
