"""What a program gets without the CUDA toolkit and without built libraries - everything that runs no kernel - and which
build of the host module it loads."""

import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def bare_tree(tmp_path_factory):
    """The package's sources alone."""
    root = tmp_path_factory.mktemp("bare")
    for name in ("dmf_b200", "include"):
        shutil.copytree(ROOT / name, root / name, ignore=shutil.ignore_patterns("*.so", "__pycache__", ".build.lock"))
    return root


def _run(tree, code):
    env = dict(os.environ, NVCC="/nonexistent/nvcc", PYTHONPATH=str(tree), CUDA_VISIBLE_DEVICES="")
    return subprocess.run([sys.executable, "-c", code], cwd=tree, env=env, capture_output=True, text=True, timeout=300)


def test_the_harness_runs_on_cpu_without_the_libraries(bare_tree):
    res = _run(bare_tree, """
import torch
import dmf_b200
from dmf_b200 import adaln, ops
from dmf_b200.harness.model import build_dmft
assert dmf_b200.__file__.startswith({root!r})
model = build_dmft("DMFT-S/2", input_size=8, dmf_depth=8, use_logvar=False, num_classes=10, attn_func="base", qk_norm=False)
x, t = torch.randn(2, 4, 8, 8), torch.rand(2)
out = model(x, t, t, torch.zeros(2, dtype=torch.long))
x = torch.randn(5, 3).bfloat16()
assert torch.equal(adaln.gelu(x), torch.nn.functional.gelu(x, approximate="tanh"))
assert ops.launch_count == 0
ops.launch_count = 0
print("ran")
""".format(root=str(bare_tree)))
    assert res.returncode == 0 and "ran" in res.stdout, res.stderr[-2000:]
    assert not list(bare_tree.rglob("*.so"))


@pytest.mark.parametrize("change", ["torch version", "torch build", "C++ ABI", "Python"])
def test_a_host_module_built_for_another_torch_or_python_is_not_loaded(monkeypatch, change):
    import sysconfig

    import torch

    from dmf_b200 import build
    here = build.host_module()
    if change == "torch version":
        monkeypatch.setattr(torch, "__version__", "2.99.0+cu131")
    elif change == "torch build":
        monkeypatch.setattr(torch.version, "git_version", "0" * 40)
    elif change == "C++ ABI":
        monkeypatch.setattr(torch, "compiled_with_cxx11_abi", lambda now=torch.compiled_with_cxx11_abi(): not now)
    else:
        monkeypatch.setattr(sysconfig, "get_config_var", lambda name: "cpython-399-x86_64-linux-gnu")
    assert build.host_module() != here and build._host_stale()
