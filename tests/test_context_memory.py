"""A context's memory over its two pools, and its choices
(tests/cpp/context_memory.cu, host code over a model of the CUDA pools)."""
import os
import subprocess

import pytest

from cpvs_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("context_memory") / "context_memory")
    src = [os.path.join(ROOT, "tests", "cpp", "context_memory.cu"), os.path.join(build.CSRC, "timing.cu")]
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-o", exe, *src], check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("what", ["budget", "full", "pool_when_needed", "lookup_choice"])
def test_context_memory(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
