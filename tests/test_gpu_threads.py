"""Contexts scanned from several threads at once, their cache regions (and so the kernels' shared memory) of different sizes:
every call succeeds and gives the oracle's windows."""
import threading

import numpy as np
import pytest

import oracle
from ffbf_b200 import Filter, Params
from test_gpu_collect import planted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbytes", [200_000, 10_000])  # the tuned scan, and the generic one
def test_threads_with_different_tables(nbytes):
    import torch

    pats, text = planted(100, nbytes, 7)
    d = torch.from_numpy(text).cuda()
    errors = []
    start = threading.Barrier(4)

    def scans(cache_log2):
        prm = Params(20, 5, 2, 1 << cache_log2, 1 << 24)
        o = oracle.Oracle.from_params(prm)
        o.build(pats)
        want = o.scan(text)["hits"]
        with Filter(prm) as f:
            f.add_patterns(pats)
            start.wait()
            for _ in range(1500):
                try:
                    f.process_device(d.data_ptr(), text.size)
                    np.testing.assert_array_equal(f.collect().hit_offsets, want)
                except Exception as e:
                    errors.append((cache_log2, str(e)))
                    return

    threads = [threading.Thread(target=scans, args=(c,)) for c in (10, 20, 14, 20)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
