"""tests/cpp/launch_rules.cu: the tuned scan's launch sizes for lone texts and batch jobs, and the tiles that follow."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_rules(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "launch_rules")
    lib = os.path.join(ROOT, "ffbf_b200", "_lib")
    subprocess.run([nvcc, "-std=c++17", "-O2", f"-I{os.path.join(ROOT, 'include')}",
                    f"-I{os.path.join(ROOT, 'ffbf_b200', 'csrc')}", os.path.join(ROOT, "tests", "cpp", "launch_rules.cu"),
                    "-o", exe, f"-L{lib}", "-lffbf", f"-Xlinker=-rpath,{lib}", "-lcuda"], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True)
    assert r.returncode == 0, r.stdout.decode() + r.stderr.decode()
