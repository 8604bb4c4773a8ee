"""Kernels that may start before their predecessor has finished (``csrc/kernels/launch.cuh``): each waits
for it, and none promises the compiler that its arguments are unaliased or read-only memory, which would
let it load from them before the wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
TEXT = {p: re.sub(r"//[^\n]*", "", open(p).read()) for p in glob.glob(os.path.join(CSRC, "*", "*.cu*"))}


def _close(text, i, pair):
    """The index after the bracket that closes the one at i."""
    depth = 0
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return i


def _kernels():
    """name -> (parameters, body)"""
    out = {}
    for text in TEXT.values():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__|__maxnreg__)?", text):
            i = m.end()
            if m.group().endswith("__"):
                i = _close(text, text.index("(", i), "()")
            name = re.compile(r"\s*(\w+)\s*\(").match(text, i)
            lo = name.end() - 1
            hi = _close(text, lo, "()")
            body = text.index("{", hi)
            out[name.group(1)] = (text[lo:hi], text[body:_close(text, body, "{}")])
    return out


KERNELS = _kernels()
WAITING = sorted(n for n, (_, body) in KERNELS.items() if "wait_previous_kernel()" in body)


def _overlapped():
    names = set()
    for text in TEXT.values():
        for m in re.finditer(r"launch_overlapped\(", text):
            arg = text[m.end():text.index(",", text.index(",", m.end()))]
            names |= {n for n in re.findall(r"(\w+_kernel)\b", text[m.end():m.end() + 120].split("grid")[0])}
            if re.match(r"\s*kern\b", arg):
                names |= {n for n in re.findall(r"auto kern = (\w+)<", text)}
    return sorted(names)


def test_the_kernels_were_found():
    assert len(WAITING) >= 17 and {"norm_fwd_kernel", "rope_kernel", "gemm_pair_kernel", "xent_bwd_kernel"} <= set(WAITING)
    assert len(_overlapped()) >= 17


@pytest.mark.parametrize("name", _overlapped())
def test_waits_for_its_predecessor(name):
    assert name in WAITING


@pytest.mark.parametrize("name", WAITING)
def test_promises_nothing_about_its_arguments(name):
    params, body = KERNELS[name]
    assert "__restrict__" not in params
    # nor asks for the read-only path itself
    assert not re.search(r"__ldg|ld\.global\.nc", body)
