"""Hosts without a matching torch: the CUDA library builds where torch is not installed, and the package works through its Python
path where the native call module does not load."""
import importlib.util
import os
import subprocess
import sys

import pytest

ROOT = os.path.join(os.path.dirname(__file__), "..")


def test_build_without_torch(monkeypatch):
    spec = importlib.util.spec_from_file_location("wkv6_b200_build", os.path.join(ROOT, "star_rwkv6_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    assert build.native_command()[-1] == "-ldl"
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    assert build.native_command() is None
    monkeypatch.setattr(build, "NATIVE", os.path.join(ROOT, "no such file"))
    monkeypatch.setattr(build.os.path, "getmtime", lambda f: 1.0)
    assert not build._stale()


def _run(code):
    code = "import sys, warnings; warnings.simplefilter('ignore'); sys.modules['star_rwkv6_b200._native'] = None\n" + code
    return subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)


def test_import_without_the_native_module():
    r = _run("warnings.simplefilter('error', RuntimeWarning)\nimport star_rwkv6_b200")
    assert r.returncode != 0 and "_native.so does not load" in r.stderr
    r = _run("from star_rwkv6_b200 import ops\nassert ops._native.wkv6(1) is None and ops._native.with_state(1) is None")
    assert r.returncode == 0, r.stderr


@pytest.mark.gpu
def test_calls_without_the_native_module():
    r = _run("""
import torch
from star_rwkv6_b200.rwkv_kernel.torch_rwkv_kernel import RWKVKernelOperator
x = [torch.randn(2, 70, 128, device="cuda").mul(0.1).bfloat16().requires_grad_(True) for _ in range(4)]
u = torch.randn(2, 64, device="cuda", requires_grad=True)
y, _ = RWKVKernelOperator(64, 70)(*x, u)
g = torch.autograd.grad(y.float().square().sum(), (*x, u))
y1, s = RWKVKernelOperator(64, 70)(*x, u, return_state=True)
assert torch.equal(y, y1) and all(t.isfinite().all() for t in (*g, s))
""")
    assert r.returncode == 0, r.stderr
