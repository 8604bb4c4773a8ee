"""Pointers that 128-bit accesses cannot use are refused on the host (-2) before anything is launched;
what the kernels read or write element by element is not.  No device is touched."""
import pytest
import torch

BF16, F32 = 1, 0


@pytest.fixture(scope="module")
def lib():
    from flextrain_b200.ops.native import cuda_lib_available, cuda_lib
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    return cuda_lib()


@pytest.mark.parametrize("bad", ["x", "y", "cos", "sin"])
def test_rope(lib, bad):
    at = {n: 4096 + (4 if n == bad else 0) for n in ("x", "y", "cos", "sin")}
    assert lib.ft_rope(at["x"], 64, at["y"], 64, at["cos"], at["sin"], 1, 1, 64, 1, 1.0, BF16, None) == -2


@pytest.mark.parametrize("bad", [0, 1, 2])
def test_swiglu(lib, bad):
    at = [4096 + (2 if i == bad else 0) for i in range(3)]
    if bad < 2:
        assert lib.ft_swiglu_fwd(at[0], at[1], 1, 64, BF16, None) == -2
    assert lib.ft_swiglu_bwd(*at, 1, 64, BF16, None) == -2


@pytest.mark.parametrize("c_dtype,align", [(BF16, 8), (F32, 4)])
@pytest.mark.parametrize("bad", ["c", "r"])
def test_gemm(lib, c_dtype, align, bad):
    c, r = 4096 + 8 * (bad == "c"), 8192 + 8 * (bad == "r")

    def call(ldc, ldr, n):
        # a product of misaligned operands: what gets past the check is refused next (-101), here as well as on a
        # machine with a device
        return lib.ft_gemm_add(4096 + 2, 0, 64, 4096 + 2, 0, 64, c, ldc, c_dtype, 1, r, ldr, 1, n, 64, BF16, None)

    assert call(64, 64, 64) == -2
    assert call(64 + align, 64, 16) == -2
    assert call(64 + 1, 64, 64) != -2                     # rows off the boundary: element by element
    assert call(64, 64 + 1, 64) != -2
    assert call(64, 64, 8) != -2                          # fewer columns than a vector chunk


@pytest.mark.gpu
def test_a_gradient_buffer_off_the_boundary_is_added_to_by_autograd():
    from flextrain_b200.ops import functional as F
    x, dy = (torch.randn(40, 64, device="cuda").bfloat16() for _ in range(2))
    w = torch.randn(64, 64, device="cuda").bfloat16().requires_grad_()
    F.linear(x, w).backward(dy)
    want, buf = w.grad.clone(), torch.ones(64 * 64 + 1, device="cuda").bfloat16()
    w.grad = buf[1:].view(64, 64)
    F.linear(x, w).backward(dy)
    assert w.grad.data_ptr() == buf.data_ptr() + 2
    # two roundings instead of one
    assert (w.grad.double() - 1 - want.double()).norm() <= 8e-3 * want.double().norm()
    with pytest.raises(RuntimeError):
        F.linear_add(x, w, torch.zeros(40 * 64 + 1, device="cuda").bfloat16()[1:].view(40, 64))
