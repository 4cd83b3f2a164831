"""The context around failures that cannot be caused through its interface (tests/native/
ctx_checks.cu: counters set and allocations refused by the host; no GPU fault, no real wait)."""
import importlib
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checks(built_lib):
    b = importlib.import_module("fast-cuda-gpu-dbscan_gb300.build")
    out = os.path.join(HERE, "native", "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "ctx_checks")
    subprocess.run([b.nvcc(), *b.ARCH, *b.NVFLAGS, os.path.join(HERE, "native", "ctx_checks.cu"),
                    "-o", exe, "-L", b.PKG, "-lgbdbscan", "-Xlinker", "-rpath," + b.PKG], check=True)
    return exe


@pytest.mark.parametrize("name", ["expand_after_a_failed_index"])
def test_check(checks, name):
    r = subprocess.run([checks, name], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
