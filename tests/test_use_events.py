"""The events of objects' last uses go back to the contexts they came from
(tests/cpp/use_events.cu, host code alone)."""
import os
import subprocess

from cpvs_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_events_stay_with_their_context(tmp_path):
    exe = str(tmp_path / "use_events")
    src = [os.path.join(ROOT, "tests", "cpp", "use_events.cu"), os.path.join(build.CSRC, "timing.cu")]
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-o", exe, *src, "-Xcompiler", "-pthread"], check=True,
                   capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
