"""Builders for the native libraries of the package.

Capability parity: flextrain/ops/op_builder/__init__.py, cpu_adam.py, async_io.py.
``HostOpsBuilder`` holds the AVX-512 Adam, the NVMe engine and host copies;
``CudaOpsBuilder`` holds every sm_100a kernel plus the pinned pool and the
peer-memory plumbing.
"""
import glob
import os
import sys

from .builder import (BuildError, CPUOpBuilder, CSRC, CUDAOpBuilder, NATIVE_DIR, OpBuilder, cuda_home,
                      nvcc_path)


def _rel(pattern):
    return sorted(os.path.relpath(p, CSRC) for p in glob.glob(os.path.join(CSRC, pattern)))


class HostOpsBuilder(CPUOpBuilder):
    def __init__(self):
        super().__init__("ft_host", _rel("host/*.cpp"), headers=_rel("host/*.h"))


class CPUAdamBuilder(HostOpsBuilder):
    """The host library exports the Adam entry points (``ft_adam_*``)."""


class AsyncIOBuilder(HostOpsBuilder):
    """The host library exports the NVMe engine entry points (``ft_nvme_*``)."""


class CudaOpsBuilder(CUDAOpBuilder):
    def __init__(self):
        super().__init__("ft_cuda", _rel("kernels/*.cu") + _rel("comm/*.cu"),
                         headers=_rel("kernels/*.cuh") + _rel("comm/*.cuh") + _rel("kernels/*.h"))


class TorchOpsBuilder(OpBuilder):
    """The autograd bindings of the kernels (``csrc/torch``): a Python extension module that uses
    PyTorch's C++ API and calls the C entry points of ``ft_cuda``, which must be loaded first."""

    kind = "torch"

    def __init__(self):
        super().__init__("ft_torch", _rel("torch/*.cpp"))

    def installed_at(self):
        import sysconfig
        import torch
        return {"torch": os.path.dirname(torch.__file__), "python": sysconfig.get_paths()["include"],
                "cuda": os.path.join(cuda_home() or "/usr/local/cuda", "include")}

    def can_build(self):
        at = self.installed_at()
        return super().can_build() and all(map(os.path.exists, (
            os.path.join(at["torch"], "include", "torch", "extension.h"), os.path.join(at["python"], "Python.h"),
            os.path.join(at["cuda"], "cuda_runtime_api.h"))))

    def compile_cmd(self, src, obj):
        import sysconfig
        import torch
        at = self.installed_at()
        dirs = [os.path.join(at["torch"], "include"),
                os.path.join(at["torch"], "include", "torch", "csrc", "api", "include"), at["python"], at["cuda"]]
        return [self.compiler(), "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall",
                f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                f"-DTORCH_EXTENSION_NAME={self.name}", f"-DFT_TORCH_VERSION={torch.__version__}",
                f"-DFT_PYTHON_ABI={sysconfig.get_config_var('SOABI')}",
                f"-I{CSRC}", *(f"-isystem{d}" for d in dirs), "-c", src, "-o", obj]

    def link_cmd(self, objs, out):
        import torch
        lib = os.path.join(os.path.dirname(torch.__file__), "lib")
        return [self.compiler(), "-shared", *objs, "-o", out, f"-L{lib}", "-ltorch", "-ltorch_cpu", "-lc10",
                "-lc10_cuda", "-ltorch_python"]

    def load_module(self):
        """The extension module, built first if it is missing or stale (and can be built)."""
        import importlib.machinery
        import importlib.util
        if self.name not in sys.modules:
            self.prepare()
            loader = importlib.machinery.ExtensionFileLoader(self.name, self.lib_path)
            spec = importlib.util.spec_from_file_location(self.name, self.lib_path, loader=loader)
            module = importlib.util.module_from_spec(spec)
            loader.exec_module(module)
            sys.modules[self.name] = module
        return sys.modules[self.name]


ALL_OPS = {"ft_host": HostOpsBuilder, "ft_cuda": CudaOpsBuilder}      # the libraries with a C ABI


def build_all(force=False, verbose=False):
    paths = []
    for cls in (*ALL_OPS.values(), TorchOpsBuilder):
        paths.append(cls().build(force=force, verbose=verbose))
    return paths
