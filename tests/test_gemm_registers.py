"""The pair kernel keeps its values in registers: one that calls a function of the divided tiles spills what lives across
the call, and the loop over whole tiles, which most products consist of, loads it again for every tile."""
import re
import subprocess

import pytest

SOURCE = """
#include "kernels/gemm2_kernel.cuh"
namespace ft { namespace gemm {
#define KERNEL(MODE, TN) \\
  template __global__ void gemm_pair_kernel<__nv_bfloat16, false, false, MODE, false, TN>( \\
      const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, void*, int64_t, int, int, int, int*, \\
      const __grid_constant__ GatherArgs);
KERNEL(kStore16, 256) KERNEL(kAcc16, 256) KERNEL(kStore32, 256) KERNEL(kAcc32, 256) KERNEL(kAcc16, 128)
} }
"""


def test_no_spills(tmp_path):
    from flextrain_b200.ops.op_builder import CudaOpsBuilder, nvcc_path
    if nvcc_path() is None:
        pytest.skip("needs nvcc")
    src = tmp_path / "pair.cu"
    src.write_text(SOURCE)
    run = subprocess.run(CudaOpsBuilder().compile_cmd(str(src), str(tmp_path / "pair.o")) + ["-Xptxas", "-v"],
                         capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stderr[-2000:]
    found = re.findall(r"Compiling entry function '(\w*gemm_pair_kernel\w*)'.*?(\d+) bytes spill stores, (\d+) bytes",
                       run.stdout + run.stderr, re.S)
    assert len(found) == 5
    # one register's worth is what the bound on registers may cost a variant; the calls cost 17 to 23
    assert all(int(stores) <= 4 for _, stores, _ in found), found
