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
    """Runs a check program, built on first use."""
    b = importlib.import_module("fast-cuda-gpu-dbscan_gb300.build")
    out = os.path.join(HERE, "native", "_build")
    os.makedirs(out, exist_ok=True)
    built = set()

    def run(prog, *args):
        exe = os.path.join(out, prog)
        if prog not in built:
            subprocess.run([b.nvcc(), *b.ARCH, *b.NVFLAGS, os.path.join(HERE, "native", prog + ".cu"),
                            "-o", exe, "-L", b.PKG, "-lgbdbscan", "-Xlinker", "-rpath," + b.PKG],
                           check=True)
            built.add(prog)
        r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr

    return run


@pytest.mark.parametrize("name", ["expand_after_a_failed_index", "a_small_run_gives_up",
                                  "a_small_run_after_a_large_one",
                                  "kept_sizes_do_not_refuse_a_run",
                                  "buffers_by_the_counted_cells",
                                  "server_estimate"])
def test_context(checks, name):
    checks("ctx_checks", name)


def test_noalloc_call_gives_up(checks):
    checks("noalloc_checks")
