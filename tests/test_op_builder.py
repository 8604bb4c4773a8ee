"""The extension module with the autograd nodes loads where it cannot be built, and its signature does not
depend on where PyTorch, Python and CUDA are installed."""
import subprocess
import sys

import pytest

from flextrain_b200.ops.op_builder import BuildError, TorchOpsBuilder

SCRIPT = """
import sys
sys.path.insert(0, {repo!r})
from flextrain_b200.ops.native import cuda_lib
from flextrain_b200.ops.op_builder import BuildError, TorchOpsBuilder
cuda_lib()
def no_compiler(self):
    raise BuildError("no compiler")
TorchOpsBuilder.{missing}
TorchOpsBuilder.is_current = lambda self: False
def build(self, *a, **k):
    raise AssertionError("tried to build")
TorchOpsBuilder.build = build
assert hasattr(TorchOpsBuilder().load_module(), "linear")
"""


@pytest.fixture(scope="module", autouse=True)
def built():
    TorchOpsBuilder().build()


@pytest.mark.parametrize("missing", ["compiler = no_compiler",
                                     "installed_at = lambda self: dict.fromkeys(('torch', 'python', 'cuda'), '/nowhere')"])
def test_a_stale_module_is_used_where_nothing_can_be_built(missing):
    from flextrain_b200.ops.op_builder.builder import REPO_ROOT
    run = subprocess.run([sys.executable, "-c", SCRIPT.format(repo=REPO_ROOT, missing=missing)], capture_output=True,
                         text=True, timeout=120)
    assert run.returncode == 0, run.stderr


def test_a_missing_module_that_cannot_be_built_is_an_error(monkeypatch, tmp_path):
    def no_compiler(self):
        raise BuildError("no compiler")
    monkeypatch.setattr(TorchOpsBuilder, "compiler", no_compiler)
    monkeypatch.setattr(TorchOpsBuilder, "lib_path", str(tmp_path / "libft_torch.so"))
    monkeypatch.delitem(sys.modules, "ft_torch", raising=False)
    with pytest.raises(BuildError):
        TorchOpsBuilder().load_module()


def test_signature_names_versions_and_no_places(monkeypatch):
    import torch
    here = TorchOpsBuilder()
    want = here.signature()
    cmd = here.compile_cmd

    def elsewhere(src, obj):
        out = cmd(src, obj)
        for name, path in installed.items():
            out = [c.replace(path, f"/opt/{name}") for c in out]
        return out

    installed = here.installed_at()
    moved = TorchOpsBuilder()
    monkeypatch.setattr(moved, "compile_cmd", elsewhere)
    monkeypatch.setattr(moved, "installed_at", lambda: {n: f"/opt/{n}" for n in installed})
    link = here.link_cmd
    monkeypatch.setattr(moved, "link_cmd", lambda objs, out: [c.replace(installed["torch"], "/opt/torch") for c in link(objs, out)])
    assert moved.signature() == want
    monkeypatch.setattr(torch, "__version__", "0.0")
    assert TorchOpsBuilder().signature() != want
