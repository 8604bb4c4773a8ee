"""The C++ autograd nodes on the CPU, over host stand-ins of the kernels (``native/host_kernels.cpp``):
buffers, layouts and autograd, which need no GPU to go wrong.  One child process runs all the cases of
``_torch_ops_worker.py``, because the stand-ins must come before ``libft_cuda.so`` in it."""
import json
import os
import subprocess
import sys

import pytest

from _torch_ops_worker import HERE, NAMES


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    from flextrain_b200.ops.op_builder import TorchOpsBuilder
    d = tmp_path_factory.mktemp("stubs")
    builder = TorchOpsBuilder()
    lib, obj = str(d / "libhost_kernels.so"), str(d / "host_kernels.o")
    subprocess.run(builder.compile_cmd(os.path.join(HERE, "native", "host_kernels.cpp"), obj), check=True)
    subprocess.run(builder.link_cmd([obj], lib), check=True)
    out = str(d / "out.json")
    run = subprocess.run([sys.executable, os.path.join(HERE, "_torch_ops_worker.py"), lib, out], capture_output=True,
                         text=True, timeout=300)
    assert run.returncode == 0, run.stderr
    with open(out) as f:
        return json.load(f)


@pytest.mark.parametrize("name", NAMES)
def test_nodes(results, name):
    assert results[name] == ""
