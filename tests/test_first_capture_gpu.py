"""A process whose first launches of the norm kernels, forward and backward, are captured into a graph."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys
sys.path.insert(0, {repo!r})
import torch
from flextrain_b200.ops import functional as F
x, w, b, dy = (torch.randn(*s, device="cuda").bfloat16() for s in ((300, 1600), (1600,), (1600,), (300, 1600)))
ins = [t.requires_grad_() for t in (x, w, b)]
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = F.layernorm(*ins, 1e-5)
    got = torch.autograd.grad(y, ins, dy)
graph.replay()
torch.cuda.synchronize()
z = F.layernorm(*ins, 1e-5)
want = torch.autograd.grad(z, ins, dy)
assert torch.equal(y, z)
assert all(torch.equal(a, c) for a, c in zip(got, want))
print("captured")
"""


def test_norm_forward_and_backward():
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", SCRIPT.format(repo=repo)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "captured" in run.stdout, run.stderr[-3000:]
