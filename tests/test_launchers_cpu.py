"""The launchers' host code over a runtime that launches nothing (``native/host_runtime.cpp``): dynamic
shared memory is granted on every device, and a first call asks for nothing that a stream capture refuses."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
BF16 = 1
OBJECTS = ("gpt_ops.cu", "gemm_tcgen05.cu", "attention.cu")
AT = [1 << 20 << i for i in range(16)]                    # addresses that nothing reads


@pytest.fixture(scope="module")
def make(tmp_path_factory):
    from flextrain_b200.ops.op_builder import CudaOpsBuilder, HostOpsBuilder, cuda_home, nvcc_path
    from flextrain_b200.ops.op_builder.builder import NATIVE_DIR
    if nvcc_path() is None:
        pytest.skip("needs nvcc for the kernels' objects")
    cuda, d, objs = CudaOpsBuilder(), tmp_path_factory.mktemp("runtime"), []
    cuda.build()
    for name in OBJECTS:
        obj = os.path.join(NATIVE_DIR, "obj", "ft_cuda", name + ".o")
        if not os.path.exists(obj):                       # the library came without them
            obj = str(d / (name + ".o"))
            (src,) = (s for s in cuda.sources if s.endswith("/" + name))
            subprocess.run(cuda.compile_cmd(src, obj), check=True)
        objs.append(obj)
    cxx, count = HostOpsBuilder().compiler(), iter(range(100))

    def new():
        """A process's state is in the library: every test loads a copy of its own."""
        lib = str(d / f"libruntime{next(count)}.so")
        subprocess.run([cxx, "-shared", "-fPIC", "-O1", "-Wl,-Bsymbolic", f"-I{cuda_home()}/include",
                        os.path.join(HERE, "native", "host_runtime.cpp"), *objs, "-o", lib], check=True)
        return ctypes.CDLL(lib)

    return new


L, F, I = ctypes.c_int64, ctypes.c_float, ctypes.c_int     # noqa: E741


def P(i):
    return ctypes.c_void_p(AT[i])


NULL = ctypes.c_void_p(None)


def norm_backward(lib, h):
    return lib.ft_norm_bwd_into(P(0), P(1), P(2), NULL, NULL, P(3), P(4), NULL, P(5), NULL, P(6), NULL, L(300), I(h), I(0),
                                I(0), I(BF16), NULL)


def product(lib, m, n):
    return lib.ft_gemm_bias(P(0), I(0), L(64), P(1), I(0), L(64), P(2), L(n), I(BF16), I(0), NULL, L(0), NULL, I(m),
                            I(n), I(64), I(BF16), NULL)


def gate(lib):
    return lib.ft_gemm_swiglu(P(0), L(64), P(1), L(64), P(2), L(128), NULL, L(256), I(256), I(128), I(64), I(BF16), NULL)


def attention(lib, d):
    return lib.ft_attn_fwd(P(0), L(d), P(1), L(d), P(2), L(d), P(3), P(4), I(1), I(128), I(1), I(1), I(d), F(1), I(BF16),
                           NULL)


def attention_backward(lib, d):
    return lib.ft_attn_bwd(P(0), L(d), P(1), L(d), P(2), L(d), P(3), P(4), L(d), P(5), P(6), P(7), P(8), L(d), P(9), L(d),
                           P(10), L(d), I(1), I(128), I(1), I(1), I(d), F(1), I(BF16), NULL)


CALLS = {f"norm_backward_{h}": (norm_backward, h) for h in (4096, 5120, 8192, 16384)}
CALLS.update(product_rows_100=(product, 100, 64), product_rows_300=(product, 300, 64), gate=(gate,))
CALLS.update({f"{f.__name__}_{d}": (f, d) for f in (attention, attention_backward) for d in (64, 128)})


@pytest.mark.parametrize("name", CALLS)
def test_every_device_grants_the_shared_memory(make, name):
    lib, (call, *args) = make(), CALLS[name]
    for dev in (0, 1, 0, 1):
        lib.host_use_device(dev)
        before = lib.host_launches()
        assert call(lib, *args) == 0, f"device {dev}"
        assert lib.host_launches() > before


@pytest.mark.parametrize("name", CALLS)
def test_a_first_call_may_be_captured(make, name):
    lib, (call, *args) = make(), CALLS[name]
    lib.host_capture(1)
    assert call(lib, *args) == 0
    assert lib.host_refused_in_capture() == 0
    assert lib.host_launches() > 0


def test_a_product_that_would_be_divided_asks_for_its_workspace(make):
    lib = make()
    lib.ft_gemm_ws_bytes.restype = L

    def call(m, n, k, ws, nbytes):
        return lib.ft_gemm_ws(P(0), I(0), L(k), P(1), I(0), L(k), P(2), L(n), I(BF16), I(0), NULL, L(0), NULL, I(m), I(n),
                              I(k), I(BF16), ws, L(nbytes), NULL)

    for m, n, k, divided in ((1024, 768, 50304, True), (1024, 768, 64, False), (100, 768, 50304, False)):
        before, nbytes = lib.host_launches(), lib.ft_gemm_ws_bytes(I(m), I(n), I(k), I(BF16))
        assert (nbytes > 0) == divided
        assert call(m, n, k, NULL, -1) == (-5 if divided else 0)
        assert lib.ft_gemm_try(P(0), I(0), L(k), P(1), I(0), L(k), P(2), L(n), I(BF16), I(0), I(m), I(n), I(k), I(BF16),
                               NULL) == (-5 if divided else 0)
        assert lib.host_launches() == before + 2 * (not divided)
        assert call(m, n, k, NULL, 0) == 0 and call(m, n, k, P(3), nbytes) == 0
        assert lib.host_launches() == before + 2 + 2 * (not divided)


@pytest.mark.parametrize("act", [0, 1])
def test_bias_rows_of_any_width_keep_their_threads_busy(make, act):
    """A thread takes eight values of one row or of several: never many more threads than that needs."""
    lib = make()
    lib.host_last_threads.restype = L
    for rows in (1, 33, 4096, 65536, 1 << 20):
        for n in (8, 16, 24, 64, 96, 248, 256, 264, 768, 6400):
            assert lib.ft_bias_act_fwd(P(0), P(1), P(2), L(rows), I(n), I(act), I(BF16), NULL) == 0
            vectors = rows * n // 8
            assert lib.host_last_threads() <= 2 * vectors + 256 * (1 + n // 256), (rows, n)
    before = lib.host_launches()                          # more row blocks than a grid's second dimension holds
    assert lib.ft_bias_act_fwd(P(0), P(1), P(2), L(2 * 65535 * 32 + 1), I(256), I(act), I(BF16), NULL) == 0
    assert lib.host_launches() == before + 3
