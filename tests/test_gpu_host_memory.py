"""tests/cpp/host_memory.cpp: a host allocation that fails inside an entry point becomes a status, not an exception."""
import subprocess

import pytest

from test_gpu_scan_errors import build_cpp

pytestmark = pytest.mark.gpu


def test_host_memory_that_runs_out_is_a_status(tmp_path):
    r = subprocess.run([build_cpp("host_memory", tmp_path, ".cpp")], capture_output=True, timeout=300)
    assert r.returncode == 0, r.stdout.decode() + r.stderr.decode()
