"""The product's C entries where no device is visible: an error code or "no workspace", and a process that lives."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import sys
sys.path.insert(0, %r)
from flextrain_b200.ops.native import cuda_lib
lib, at, bf16 = cuda_lib(), [1 << 20 << i for i in range(5)], 1
rc = {
    "ws_bytes": lib.ft_gemm_ws_bytes(1024, 768, 50304, bf16),
    "plan": lib.ft_gemm_split_plan(1024, 768, 50304, bf16, 0) - 256,
    "tile_n": lib.ft_gemm_tile_n(1024, 768, bf16, 0) - 256,
    "product": lib.ft_gemm(at[0], 0, 64, at[1], 0, 64, at[2], 768, bf16, 0, 1024, 768, 64, bf16, None),
    "workspace": lib.ft_gemm_ws(at[0], 0, 50304, at[1], 0, 50304, at[2], 768, bf16, 0, None, 0, None, 1024, 768, 50304,
                                bf16, at[3], 1 << 30, None),
    "gradients": lib.ft_gemm_dw_db(at[0], 768, at[1], 768, at[2], 768, 0, at[3], 0, 1024, 768, 768, bf16, None),
    "gate": lib.ft_gemm_swiglu(at[0], 64, at[1], 64, at[2], 128, None, 0, 256, 128, 64, bf16, None),
}
wrong = [n for n, v in rc.items() if (v == 0) != (n in ("ws_bytes", "plan", "tile_n"))]
print("ended", wrong, rc)
""" % ROOT


def test_no_entry_ends_the_process():
    from flextrain_b200.ops.native import cuda_lib_available
    if not cuda_lib_available():
        pytest.skip("the CUDA library is not built")
    run = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300,
                         env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert run.returncode == 0 and "ended []" in run.stdout, (run.returncode, run.stdout, run.stderr[-2000:])
