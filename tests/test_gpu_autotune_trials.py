"""tests/cpp/autotune_trials.cu: the batch autotuner times the launches that a batch makes."""
import subprocess

import pytest

from test_gpu_scan_errors import build_cpp

pytestmark = pytest.mark.gpu


def test_trials_run_as_the_batch_does(tmp_path):
    r = subprocess.run([build_cpp("autotune_trials", tmp_path)], capture_output=True, timeout=300)
    assert r.returncode == 0, r.stdout.decode() + r.stderr.decode()
