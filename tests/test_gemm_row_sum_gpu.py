"""Weight and bias gradient of a projection in one product: the sums of dy's columns against exact ones (small
integers: fp32 sums are exact, a 16-bit result is the exact one rounded once), where the product sums on the way
(tiles of up to 128 columns) and where the sum is a pass of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one tile, tiles of 64 and 128 columns in one and in two columns, ragged rows and reduction, more tiles than pairs (a pair takes one
# of the first column after another tile), and two that do not sum
@pytest.mark.parametrize("t,n,k,inside", [(64, 256, 64, True), (200, 304, 264, True), (136, 768, 768, True),
                                          (2048, 2304, 768, True), (1, 136, 136, True), (136, 6400, 640, True),
                                          (72, 4096, 4096, False),
                                          (72, 128, 256, False)])
@pytest.mark.parametrize("held", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gradients(t, n, k, inside, held, dtype):
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(t + n)
    ints = lambda *s: torch.randint(-2, 3, s, generator=gen, device="cuda").to(dtype)              # noqa: E731
    x, w, b, dy = ints(t, k), ints(n, k).requires_grad_(), ints(n).requires_grad_(), ints(t, n)
    if held:
        w.grad, b.grad = ints(n, k), ints(n)
    base = [0 if p.grad is None else p.grad.double() for p in (w, b)]
    assert (n > 128 and cuda_lib().ft_gemm_tile_n(n, k, 1, 74) <= 128) == inside
    y = ops.linear_bias(x, w, b)
    y.backward(dy)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    assert torch.equal(w.grad, (base[0] + dy.double().T @ x.double()).to(dtype))
    assert torch.equal(b.grad, (base[1] + dy.double().sum(0)).to(dtype))
