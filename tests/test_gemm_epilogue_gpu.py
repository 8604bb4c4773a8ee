"""The GEMM epilogue's addend pipeline (chunks of 16 columns requested ahead of the accumulator) at
the places where it can go wrong: a last chunk, tile or row block that is not full, row strides that
rule 16-byte access out, several tiles per CTA, an addend that is C itself and one that is not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (m, n): one row block of either kernel and its edges; n around the 16-column chunk and the
# 256-column tile; the last shape gives every CTA pair several tiles
@pytest.mark.parametrize("m,n", [(1, 8), (128, 256), (129, 248), (300, 264), (257, 777), (40, 1000), (6000, 2568)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("in_place", [True, False])
def test_addend_is_added_exactly_once(m, n, out_dtype, in_place):
    from flextrain_b200.ops.cuda_ops import gemm
    from flextrain_b200.ops.native import cuda_lib
    k, dev = 64, torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(m + n)
    # integers up to 8 with 64 terms: every product sum and addend is exact in fp32, and in bf16 the
    # result is the exact sum rounded once
    a, b = (torch.randint(-3, 4, (r, k), generator=gen, device=dev).to(torch.bfloat16) for r in (m, n))
    rows = torch.randint(-100, 101, (m + 2, n), generator=gen, device=dev).to(out_dtype)
    out = rows.clone()
    if in_place:
        gemm(a, False, b, False, m, n, k, out=out[1:-1], accumulate=True)
    else:
        gemm(a, False, b, False, m, n, k, out=out[1:-1], add=rows[1:-1])
    want = rows.clone()
    want[1:-1] = (rows[1:-1].double() + a.double() @ b.double().T).to(out_dtype)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    assert torch.equal(out, want)                        # the rows around the output too
