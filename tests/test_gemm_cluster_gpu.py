"""The GEMM of few tiles (csrc/kernels/gemm_cluster.cuh): the sizes below take each of its tile widths and the divided
reduction, with rows, columns and reductions that end inside a tile, outputs and addends that are columns of wider
matrices, and every operand layout and epilogue.  Small integers: every sum is exact in fp32, a 16-bit result is
the exact one rounded once."""
import pytest
import torch

# rows, columns, reduction -> tile width, pairs a cluster (without an addend)
SHAPES = {(129, 8, 72): (64, 1), (304, 264, 520): (64, 1), (257, 72, 3080): (128, 2),
          (256, 384, 3080): (128, 2), (2800, 264, 3080): (128, 2), (2047, 768, 8): (128, 1),
          (3000, 768, 1032): (128, 1), (1000, 3080, 200): (192, 1), (3000, 776, 3080): (192, 1),
          (2047, 2304, 520): (256, 1), (2048, 2304, 136): (256, 1)}
# the same with an addend, where the rule answers otherwise; tiles of 192 columns take one only where the reduction is long
ADDED = {(1000, 3080, 200): (256, 1), (3000, 776, 3080): (256, 1), (520, 3104, 5480): (192, 1)}


def _plan(m, n, k, acc=0, pairs=74):
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    p = cuda_lib().ft_gemm_cluster_plan(m, n, k, acc, pairs)
    return p & 0xffff, p >> 16


@pytest.mark.parametrize("shape,plan", SHAPES.items())
def test_the_shapes_take_every_kernel(shape, plan):
    assert _plan(*shape) == plan
    assert _plan(*shape, acc=1) == ADDED.get(shape, plan)


def test_the_shapes_take_every_kernel_that_adds():
    assert {_plan(*s, acc=1) for s in [*SHAPES, *ADDED]} == {(64, 1), (128, 1), (128, 2), (192, 1), (256, 1)}
    assert all(_plan(*s, acc=1) == plan for s, plan in ADDED.items())


def test_the_rule_leaves_large_products_alone():
    assert {p[0] for p in SHAPES.values()} == {64, 128, 192, 256} and (128, 2) in SHAPES.values()
    for m, n, k in ((4096, 4096, 4096), (256, 50304, 768), (256, 256, 50304), (192, 12288, 4096)):
        assert _plan(m, n, k) == (0, 0)
    assert _plan(256, 256, 256, pairs=0) == (0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", list(dict.fromkeys([*SHAPES, *ADDED])))
@pytest.mark.parametrize("layout", ["fwd", "dgrad", "wgrad"])
@pytest.mark.parametrize("mode", ["store", "add", "accumulate", "bias", "bias_add"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_products(shape, layout, mode, dtype):
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    m, n, k = shape
    a_mn, b_mn = layout == "wgrad", layout != "fwd"
    if mode.startswith("bias") and layout != "fwd":
        pytest.skip("the bias belongs to the forward product")
    if a_mn and m % 8:
        pytest.skip("rows of this operand are not 16-byte aligned")
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    ints = lambda hi, *s: torch.randint(-hi, hi + 1, s, generator=gen, device="cuda").to(dtype)      # noqa: E731
    a, b, bias = ints(1, m, k), ints(1, n, k), ints(9, n)
    ld = (n + 7) // 8 * 8 + 8
    held, addend = ints(50, m + 2, ld), ints(50, m + 2, ld)
    at = (slice(1, -1), slice(8, 8 + n) if n % 8 == 0 and ld >= n + 8 else slice(0, n))
    prod, out = a.double() @ b.double().T, held.clone()
    if mode.startswith("bias"):
        res = addend[at] if mode == "bias_add" else None
        out[at] = ops.linear_bias(a, b, bias, res)
        want = prod + bias.double() + (0 if res is None else res.double())
    else:
        A, B = (t.t().contiguous() if mn else t for t, mn in ((a, a_mn), (b, b_mn)))
        add = addend[at] if mode == "add" else None
        ops.gemm(A, a_mn, B, b_mn, m, n, k, out=out[at], accumulate=mode == "accumulate", add=add)
        want = prod + (addend[at].double() if mode == "add" else held[at].double() if mode == "accumulate" else 0)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    expect = held.clone()
    expect[at] = want.to(dtype)
    assert torch.equal(out, expect)


# outputs whose rows end between units of eight, which the copy engine would write to their end: the other kernels' work
@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 7, 63, 65, 129, 259])
@pytest.mark.parametrize("accumulate", [False, True])
def test_odd_widths(n, accumulate):
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(n)
    ints = lambda hi, *s: torch.randint(-hi, hi + 1, s, generator=gen, device="cuda").bfloat16()     # noqa: E731
    m, k = 300, 136
    a, b, held = ints(2, m, k), ints(2, n, k), ints(50, m + 2, (n + 7) // 8 * 8 + 8)
    out = held.clone()
    ops.gemm(a, False, b, False, m, n, k, out=out[1:-1, :n], accumulate=accumulate)
    want = held.clone()
    want[1:-1, :n] = (a.double() @ b.double().T + (held[1:-1, :n].double() if accumulate else 0)).bfloat16()
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    assert torch.equal(out, want)


# rows of the weight (the tiles' rows), its columns, tokens -> tile width, pairs a cluster: each width that sums, whole and divided, several
# columns of tiles
ROW_SUMS = {(136, 136, 64): (64, 1), (264, 72, 200): (64, 1), (768, 776, 1032): (64, 1), (1032, 264, 2048): (128, 2),
            (304, 2304, 136): (64, 1), (2304, 768, 520): (128, 1), (528, 3144, 64): (192, 1), (776, 2512, 72): (192, 1)}


def test_the_row_sums_take_every_kernel():
    assert set(ROW_SUMS.values()) == {(64, 1), (128, 1), (128, 2), (192, 1)}
    for shape, plan in ROW_SUMS.items():
        assert [_plan(*shape, acc=2 + held) for held in (0, 1)] == [plan, plan]


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,t", ROW_SUMS)
@pytest.mark.parametrize("held", [False, True])
def test_row_sums(n, k, t, held):
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(n + t)
    ints = lambda *s: torch.randint(-1, 2, s, generator=gen, device="cuda").bfloat16()              # noqa: E731
    x, w, b, dy = ints(t, k), ints(n, k).requires_grad_(), ints(n).requires_grad_(), ints(t, n)
    if held:
        w.grad, b.grad = ints(n, k), ints(n)
    base = [0 if p.grad is None else p.grad.double() for p in (w, b)]
    ops.linear_bias(x, w, b).backward(dy)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    assert torch.equal(w.grad, (base[0] + dy.double().T @ x.double()).bfloat16())
    assert torch.equal(b.grad, (base[1] + dy.double().sum(0)).bfloat16())


# tokens, rows and columns of the weight -> tile width and pairs a cluster of both products of a projection's backward in one launch,
# without and with the bias gradient; (0, 0): one launch each
BACKWARD = {(136, 136, 8): ((64, 1), (64, 1)), (304, 264, 520): ((64, 1), (64, 1)), (1000, 776, 768): ((128, 1), (128, 1)),
            (256, 2304, 768): ((128, 2), (128, 2)), (300, 2304, 768): ((128, 2), (128, 2)), (2000, 264, 264): ((128, 2), (128, 2)),
            (2048, 2304, 768): ((256, 1), (192, 1)), (1000, 1032, 1544): ((256, 1), (0, 0)), (1024, 2304, 768): ((0, 0), (0, 0))}


def test_the_backward_shapes_take_every_kernel():
    from flextrain_b200.ops.native import cuda_lib, cuda_lib_available
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    lib = cuda_lib()
    for (t, n, k), plans in BACKWARD.items():
        got = [lib.ft_gemm_backward_plan(t, n, k, 1, sums, 74) for sums in (0, 1)]
        assert tuple((p & 0xffff, p >> 16) for p in got) == plans
    assert {p for plans in BACKWARD.values() for p in plans} == {(0, 0), (64, 1), (128, 1), (128, 2), (192, 1), (256, 1)}
    for t, n, k in ((128, 4096, 256), (4096, 128, 256), (4096, 4096, 4096), (64, 64, 64)):
        assert lib.ft_gemm_backward_plan(t, n, k, 0, 0, 74) == 0
    assert lib.ft_gemm_backward_plan(256, 256, 256, 0, 0, 0) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("t,n,k", BACKWARD)
@pytest.mark.parametrize("held", [False, True])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_both_products_of_a_backward(t, n, k, held, bias, dtype):
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(t + n)
    ints = lambda *s: torch.randint(-1, 2, s, generator=gen, device="cuda").to(dtype)              # noqa: E731
    x, w, b, dy = ints(t, k).requires_grad_(), ints(n, k).requires_grad_(), ints(n).requires_grad_(), ints(t, n)
    if held:
        w.grad, b.grad = ints(n, k), ints(n)
    base = [0 if p.grad is None else p.grad.double() for p in (w, b)]
    y = ops.linear_bias(x, w, b) if bias else ops.linear(x, w)
    before = cuda_lib().ft_launch_count()
    y.backward(dy)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    plan = BACKWARD[t, n, k][bias]
    assert (cuda_lib().ft_launch_count() - before == 1) == (plan != (0, 0))
    assert torch.equal(x.grad, (dy.double() @ w.detach().double()).to(dtype))
    assert torch.equal(w.grad, (base[0] + dy.double().T @ x.detach().double()).to(dtype))
    if bias:
        assert torch.equal(b.grad, (base[1] + dy.double().sum(0)).to(dtype))


@pytest.mark.gpu
def test_launches_in_a_row_and_on_two_streams():
    """Each launch sets itself up under the one before it, and shares the SMs with one of another stream."""
    from flextrain_b200.ops import cuda_ops as ops
    from flextrain_b200.ops.native import cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(3)
    ints = lambda *s: torch.randint(-1, 2, s, generator=gen, device="cuda").bfloat16()              # noqa: E731
    shapes = [(512, 512, 512), (256, 1024, 512), (1000, 512, 512), (512, 512, 3072), (2048, 768, 512)]
    work = [(ints(m, k), ints(n, k), torch.zeros(m, n, dtype=torch.bfloat16, device="cuda"), m, n, k) for m, n, k in shapes]
    want = [(a.double() @ b.double().T) for a, b, *_ in work]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[w[2].clone() for w in work] for _ in streams]
    torch.cuda.synchronize()
    for _ in range(3):
        for s, out in zip(streams, outs):
            with torch.cuda.stream(s):
                for (a, b, _, m, n, k), c in zip(work, out):
                    ops.gemm(a, False, b, False, m, n, k, out=c)
    torch.cuda.synchronize()
    assert cuda_lib().ft_gemm_error() == 0
    for out in outs:
        for c, w in zip(out, want):
            assert torch.equal(c, w.bfloat16())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(300, 264, 72), (256, 384, 3080), (2047, 2304, 520)])
def test_one_row_added_to_all(m, n, k):
    """A residual whose rows are one row, as broadcasting leaves it."""
    from flextrain_b200.ops import cuda_ops as ops
    gen = torch.Generator(device="cuda").manual_seed(m)
    ints = lambda hi, *s: torch.randint(-hi, hi + 1, s, generator=gen, device="cuda").bfloat16()      # noqa: E731
    x, w, row = ints(1, m, k), ints(1, n, k), ints(50, n)
    y = ops.linear_add(x, w, row.expand(m, n))
    assert torch.equal(y, (x.double() @ w.double().T + row.double()).bfloat16())
