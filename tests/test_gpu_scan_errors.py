"""tests/cpp/scan_errors.cu: a scan whose kernel raised an error flag is never collected as a whole result."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def build_cpp(name, tmp_path, suffix=".cu"):
    """Builds tests/cpp/<name><suffix> against libffbf.so and its internal headers; returns the program's path."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / name)
    lib = os.path.join(ROOT, "ffbf_b200", "_lib")
    subprocess.run([nvcc, "-std=c++17", "-O2", f"-I{os.path.join(ROOT, 'include')}",
                    f"-I{os.path.join(ROOT, 'ffbf_b200', 'csrc')}", os.path.join(ROOT, "tests", "cpp", name + suffix),
                    "-o", exe, f"-L{lib}", "-lffbf", f"-Xlinker=-rpath,{lib}", "-lcuda"], check=True)
    return exe


def test_error_flags_of_a_scan_are_reported(tmp_path):
    r = subprocess.run([build_cpp("scan_errors", tmp_path)], capture_output=True, timeout=300)
    assert r.returncode == 0, r.stdout.decode() + r.stderr.decode()
