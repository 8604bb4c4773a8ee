"""Rotary embedding with the heads of a token split over several CTAs: head counts around the group of
four, few tokens (many ranges) and many (one range), heads beyond the rotated ones untouched."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [1, 3, 4, 5, 13, 80])
@pytest.mark.parametrize("tokens,d", [(1, 64), (37, 128), (2100, 64), (40000, 16)])
def test_rope_over_head_ranges(heads, tokens, d):
    from flextrain_b200.ops import reference as ref
    from flextrain_b200.ops.cuda_ops import rope_heads_inplace
    cos, sin = ref.rope_tables(tokens, d, 10000.0, device=torch.device("cuda"))
    x = torch.randn(1, tokens, (heads + 2) * d, device="cuda").bfloat16()
    want = x.clone().view(1, tokens, heads + 2, d)
    # both sides round one fp32 expression once; contraction may move the last bit before that
    want[:, :, :heads] = ref.rope(want[:, :, :heads].float(), cos, sin).bfloat16()
    got = rope_heads_inplace(x.clone(), cos, sin, heads, d).view_as(want)
    assert torch.equal(got[:, :, heads:], want[:, :, heads:])
    assert torch.allclose(got.float(), want.float(), rtol=2 ** -7, atol=1e-4)
