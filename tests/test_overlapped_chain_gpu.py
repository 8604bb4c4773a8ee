"""A hundred rounds of small dependent kernels over the same few buffers, launched one under the end of the
other, against the same with every launch waited for: forward chains, and a backward through all of them."""
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
gen = torch.Generator("cuda").manual_seed(1)
def r(*s, std=1.0):
    return (std * torch.randn(*s, generator=gen, device="cuda")).bfloat16()
out = []
for rows, h, heads in ((64, 256, 4), (200, 384, 6), (1000, 768, 12)):
    x, lw, lb, b3, wqkv, wo, w_gu, w_d, b = (r(2, rows, h), r(h), r(h), r(3 * h), r(3 * h, h, std=.05), r(h, h, std=.05),
                                             r(2 * 2 * h, h, std=.05), r(h, 2 * h, std=.05), r(h))
    cos, sin = F.rope_tables(rows, 64, 10000.0, device=torch.device("cuda"))
    ws = [t.requires_grad_() for t in (lw, lb, b3, wqkv, wo, w_gu, w_d, b)]
    def step(x):
        h1 = F.layernorm(x, lw, lb, 1e-5)
        qkv = F.rope_heads_inplace(F.bias_add(F.linear(h1, wqkv), b3), cos, sin, 2 * heads, 64)
        a = F.attention_packed(qkv, heads, heads, 64)
        s, n = F.add_rmsnorm(x, F.linear(a, wo), lw, 1e-5)
        g = F.bias_gelu(F.linear_add(F.swiglu(F.linear(n, w_gu)), w_d, s), b)
        return F.add_layernorm(g, s, lw, lb, 1e-5)[1]
    with torch.no_grad():
        y = x
        for _ in range(100):
            y = step(y)
    out.append(y)
    # through everything but attention, whose dQ is added up in any order
    def part(x):
        qkv = F.rope_heads_inplace(F.bias_add(F.linear(F.layernorm(x, lw, lb, 1e-5), wqkv), b3), cos, sin, 2 * heads, 64)
        s, n = F.add_rmsnorm(x, F.linear(qkv[..., :h], wo), lw, 1e-5)
        return F.bias_gelu(F.linear_add(F.swiglu(F.linear(n, w_gu)), w_d, s), b)
    y = leaf = x.clone().requires_grad_()
    for _ in range(8):
        y = part(y)
    out += [y.detach(), *torch.autograd.grad(y, [leaf, *ws], r(2, rows, h))]
torch.cuda.synchronize()
torch.save([t.cpu() for t in out], {out!r})
"""


def test_overlapped_and_serialised_launches_agree(tmp_path):
    import torch
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    got = []
    for blocking in ("0", "0", "1"):
        out = str(tmp_path / f"{len(got)}.pt")
        env = dict(os.environ, CUDA_LAUNCH_BLOCKING=blocking)
        run = subprocess.run([sys.executable, "-c", SCRIPT.format(repo=repo, out=out)], env=env, capture_output=True,
                             text=True, timeout=300)
        assert run.returncode == 0, run.stderr[-3000:]
        got.append(torch.load(out))
    for a, b, c in zip(*got):
        assert a.isfinite().all() and a.float().norm() > 0
        assert torch.equal(a, c) and torch.equal(b, c)
