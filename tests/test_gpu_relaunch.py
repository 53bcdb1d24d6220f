"""A prepared batch launched again after its contexts were used alone: every job's results are those of its own text."""
import numpy as np
import pytest

from ffbf_b200 import Batch, Filter
from test_gpu_collect import PRM, check, planted

pytestmark = pytest.mark.gpu


def clear(f):
    import torch
    f.clear_ff()
    torch.cuda.synchronize()


@pytest.mark.parametrize("n_hits,nbytes,newline", [
    (2000, 300_000, 80),           # more windows than the batch has room for
    (300, 3 << 20, 3_000_000),     # lines over more tiles than the single launch walks
    (12_000, 70 << 20, 80),        # a text whose tiles are 16 KiB at least
])
def test_plain_scans_between_launches(n_hits, nbytes, newline):
    """Newline tiles follow a scan's rows per stream: those of the scans in between are not the batch's."""
    import torch

    pats, text = planted(n_hits, nbytes, 41 + n_hits, newline)
    others = [planted(40, n, 5)[1] for n in (200_003, 30_000, 9 << 20)]
    d = torch.from_numpy(text).cuda()
    with Filter(PRM) as f, Batch() as b:
        f.add_patterns(pats)
        b.add(f, d.data_ptr(), text.size)
        b.prepare()
        for other in others:
            t = torch.from_numpy(other).cuda()
            f.process_device(t.data_ptr(), other.size)
            f.collect()
            clear(f)
            b.launch()
            b.wait()
            assert check(f, PRM, pats, text, f.collect()) >= n_hits
