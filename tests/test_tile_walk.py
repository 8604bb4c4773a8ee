"""The walk over a product's tiles (csrc/kernels/tile_walk.cuh), compiled for the host with the undefined-behaviour
checks on."""
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def build_walk(tmp):
    from flextrain_b200.ops.op_builder import HostOpsBuilder
    exe = str(tmp / "tile_walk")
    subprocess.run([HostOpsBuilder().compiler(), "-O1", "-std=c++17", "-fsanitize=undefined",
                    "-fsanitize-undefined-trap-on-error", "-I" + os.path.join(os.path.dirname(HERE), "csrc"),
                    os.path.join(HERE, "native", "tile_walk.cpp"), "-o", exe], check=True)
    return exe


def ask(exe, lines):
    """Answers to the lines, a list of tuples of numbers each."""
    run = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, f"tile_walk ended with {run.returncode}"
    return [[tuple(map(int, w.split(","))) for w in line.split()] for line in run.stdout.splitlines()]


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    return build_walk(tmp_path_factory.mktemp("walk"))


def test_every_tile_once_and_a_look_past_the_end(walk):
    rng = random.Random(3)
    # row blocks in whole groups (16, 32) and with a rest; producers look up to 74 tiles ahead
    shapes = [(mt, nt, gm) for mt in (1, 2, 15, 16, 17, 32, 64) for nt in (1, 3, 16) for gm in (1, 8, 16)]
    shapes += [(rng.randint(1, 90), rng.randint(1, 60), rng.choice([4, 16])) for _ in range(60)]
    for (mt, nt, gm), tiles in zip(shapes, ask(walk, [f"walk {m} {n} {g} 74" for m, n, g in shapes])):
        assert sorted(tiles[:mt * nt]) == [(m, n) for m in range(mt) for n in range(nt)]
        assert all(0 <= m < mt and 0 <= n < nt for m, n in tiles[mt * nt:])
