"""The pool of device buffers on the host: tests/cpp/pool_check.cpp compiles
qmb_mem.cu over a stand-in for the CUDA calls that it makes (no GPU needed)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "pool_check.cpp")


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pool") / "pool_check")
    cmd = ["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "qmbcuda_b200", "csrc"),
           "-I", "/usr/local/cuda/include", SRC, "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=60).stdout
    return dict(line.split(" ", 1) for line in out.splitlines())


@pytest.mark.parametrize("case", ["reuse", "released_after_reset", "kept_before_reset", "two_contexts", "refused_free", "trim"])
def test_pool(results, case):
    assert results[case] == "ok"
