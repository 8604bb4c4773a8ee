"""What a product issued from Python asks of the library: one call, and scratch only where it is divided."""
import pytest
import torch

BF16 = 1


class Library:
    def __init__(self, divide):
        self.divide, self.calls = divide, []

    def ft_gemm_ws_bytes(self, m, n, k, c_dtype):
        self.calls.append(("bytes", m, n, k, c_dtype))
        return 4096 if self.divide else 0

    def ft_gemm_ws(self, *args):
        assert len(args) == 20
        self.calls.append(("product", *args[13:19]))
        return -5 if self.divide and args[18] == -1 else 0

    def ft_gemm_try(self, *args):
        assert len(args) == 15
        self.calls.append(("product", *args[10:14], None, -1))
        return -5 if self.divide else 0


@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("divide", [False, True])
def test_calls_of_a_product(monkeypatch, divide, add):
    from flextrain_b200.ops import cuda_ops
    lib = Library(divide)
    monkeypatch.setattr(cuda_ops, "cuda_lib", lambda: lib)
    monkeypatch.setattr(cuda_ops, "stream_handle", lambda: None)
    a, b = torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(8, 64, dtype=torch.bfloat16)
    out = cuda_ops.gemm(a, False, b, False, 4, 8, 64, add=torch.zeros(4, 8, dtype=torch.bfloat16) if add else None)
    assert out.shape == (4, 8)
    assert [c[0] for c in lib.calls] == (["product", "bytes", "product"] if divide else ["product"])
    sizes, asked = (4, 8, 64, BF16), (None, -1)
    assert lib.calls[0] == ("product", *sizes, *asked)
    if divide:
        assert lib.calls[1] == ("bytes", 4, 8, 64, BF16)
        assert lib.calls[2][:5] == ("product", *sizes) and lib.calls[2][5] is not None and lib.calls[2][6] == 4096


def test_a_divided_product_without_memory_runs_whole(monkeypatch):
    from flextrain_b200.ops import cuda_ops
    lib = Library(True)
    monkeypatch.setattr(cuda_ops, "cuda_lib", lambda: lib)
    monkeypatch.setattr(cuda_ops, "stream_handle", lambda: None)
    a, out = torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(4, 4, dtype=torch.bfloat16)

    def refuse(*args, **kwargs):
        raise torch.OutOfMemoryError("no memory")
    monkeypatch.setattr(torch, "empty", refuse)
    cuda_ops.gemm(a, False, a, False, 4, 4, 64, out=out)
    assert lib.calls[-1][5:] == (None, 0)

