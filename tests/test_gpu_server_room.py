"""Served requests with more windows than their collection has CTAs for (one window per 2 KiB of text, at least 512), up to
the most one launch finishes and beyond: the results are the oracle's, and up to 16384 windows a request takes as many
launches as one with a few."""
import numpy as np
import pytest

import oracle
from ffbf_b200 import Filter, Server, kernel_launches
from test_gpu_collect import PRM, planted
from test_gpu_server import drain

pytestmark = pytest.mark.gpu


def test_requests_around_their_room():
    sizes = [(5, 100_000), (511, 100_001), (512, 100_002), (513, 100_003), (1024, 100_004), (1025, 100_005),
             (3000, 100_006), (2049, 4 << 20), (16384, 600_001), (16385, 600_002), (40, 100_007)]
    with Filter(PRM) as f, Server() as srv:
        pats = planted(0, 1000, 300)[0]
        f.add_patterns(pats)
        sid = srv.add_set(f)
        o = oracle.Oracle.from_params(PRM)
        o.build(pats)
        launches = {}
        for n, nbytes in sizes:
            text = planted(n, nbytes, 300)[1]
            s = o.scan(text)
            before = kernel_launches()
            rid = srv.submit(sid, text)
            r = drain(srv, 1)[rid]
            launches.setdefault(s["hits"].size <= 16384, set()).add(kernel_launches() - before)
            assert s["hits"].size >= n
            np.testing.assert_array_equal(r.hit_offsets, s["hits"])
            np.testing.assert_array_equal(r.line_start, s["line_start"])
            np.testing.assert_array_equal(r.line_end, s["line_end"])
        assert len(launches[True]) == 1 and min(launches[False]) > max(launches[True])
