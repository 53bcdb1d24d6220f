"""Scans of device texts enqueued without collecting the ones before: feed-forward bits accumulate over all of them, and
the last one's results are the ones collected. The sizes make the scans differ in CTA size, rows and items, and there are
more of them than the context keeps upload blocks for."""
import numpy as np
import pytest

import oracle
from ffbf_b200 import Filter
from test_gpu_collect import PRM, planted

pytestmark = pytest.mark.gpu


def device_texts(sizes, seed):
    import torch
    pats = planted(0, 1000, seed)[0]
    texts = [planted(n // 2000, n, seed)[1] for n in sizes]
    return pats, texts, [torch.from_numpy(t).cuda() for t in texts]


@pytest.mark.parametrize("sizes", [
    [48 << 20, 200_003, 3 << 20],
    [48 << 20] + [20_000 + 37_123 * i * i for i in range(19)],
])
def test_every_queued_scan_is_made(sizes):
    pats, texts, dev = device_texts(sizes, 71)
    o = oracle.Oracle.from_params(PRM)
    o.build(pats)
    for t in texts:
        last = o.scan(t)
    with Filter(PRM) as f:
        f.add_patterns(pats)
        f.process_device(dev[-1].data_ptr(), texts[-1].size)  # the filter's tables are built here
        f.collect()
        f.clear_ff()
        for t, d in zip(texts, dev):
            f.process_device(d.data_ptr(), t.size)
        r = f.collect()
        np.testing.assert_array_equal(r.hit_offsets, last["hits"])
        np.testing.assert_array_equal(r.line_start, last["line_start"])
        np.testing.assert_array_equal(f.get_filters()[1], o.ff)


def test_a_captured_scan_replays_its_own_text():
    import torch

    pats, texts, dev = device_texts([2 << 20, 600_000, 30_000], 72)
    o = oracle.Oracle.from_params(PRM)
    o.build(pats)
    o.scan(texts[0])
    with Filter(PRM) as f:
        f.add_patterns(pats)
        f.process_device(dev[0].data_ptr(), texts[0].size)  # buffers and tables of the captured scan
        f.collect()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(f.stream)):
            f.process_device(dev[0].data_ptr(), texts[0].size)
        for _ in range(10):
            for t, d in zip(texts[1:], dev[1:]):
                f.process_device(d.data_ptr(), t.size)
        f.collect()
        f.clear_ff()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(f.get_filters()[1], o.ff)
        del graph
