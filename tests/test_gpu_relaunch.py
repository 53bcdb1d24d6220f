"""A prepared batch launched again after its contexts were used alone: every job's results are those of its own text."""
import numpy as np
import pytest

from ffbf_b200 import Batch, Filter, Params
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


def test_wait_after_other_use_of_the_contexts():
    """A member scanned alone after the launch keeps that scan's results over the batch's wait, and a member that is gone
    is left alone; the others' results are the batch's."""
    import torch

    jobs = [planted(30 + n, 400_000 + n, 60 + n) for n in range(3)]
    other = planted(25, 90_001, 60)[1]  # shorter than the job's text
    d_other = torch.from_numpy(other).cuda()
    texts = [torch.from_numpy(t).cuda() for _, t in jobs]
    filters = [Filter(PRM) for _ in jobs]
    with Batch() as b:
        for f, (pats, text), d in zip(filters, jobs, texts):
            f.add_patterns(pats)
            b.add(f, d.data_ptr(), text.size)
        for gone in (False, True):
            for f in filters:
                clear(f)
            b.launch()
            torch.cuda.synchronize()  # the launch is done, though not waited for through the batch
            clear(filters[0])
            filters[0].process_device(d_other.data_ptr(), other.size)
            if gone:
                filters[2].close()
            b.wait()
            check(filters[0], PRM, jobs[0][0], other, filters[0].collect())
            for i in (1,) if gone else (1, 2):
                check(filters[i], PRM, *jobs[i], filters[i].collect())
    for f in filters:
        f.close()


def test_launch_after_a_segmented_scan():
    """A host text scanned in segments on a member is forgotten by the next launch: matches are those of the job's text."""
    import torch

    prm = Params(20, 5, 2, 1 << 20, 1 << 24)
    pats, text = planted(200, 24 << 20, 81)  # longer than a segment: the scan in between replaces no buffer
    long_text = planted(3000, 40 << 20, 81)[1]
    d = torch.from_numpy(text).cuda()
    with Filter(prm) as f, Batch() as b:
        f.add_patterns(pats)
        b.add(f, d.data_ptr(), text.size)
        b.prepare()
        f.set_hbm_budget(32 << 20)  # segments of about 18 MB
        check(f, prm, pats, long_text, f.process(long_text))
        clear(f)
        b.launch()
        b.wait()
        check(f, prm, pats, text, f.collect())


def test_results_over_the_shared_room():
    """A batch's jobs share their result room, which follows what a launch needed: jobs that found none are collected by
    themselves, and the next launch has room for all but those with more than 16384 windows."""
    import torch
    from ffbf_b200 import kernel_launches

    jobs = [planted(n, 600_000 + n, 90) for n in (0, 16384, 100, 9000, 511)] + [planted(16390, 600_000, 90)]
    filters = [Filter(PRM) for _ in jobs]
    texts = [torch.from_numpy(t).cuda() for _, t in jobs]
    with Batch() as b:
        for f, (pats, text), d in zip(filters, jobs, texts):
            f.add_patterns(pats)
            b.add(f, d.data_ptr(), text.size)
        for launch in range(3):
            for f in filters:
                clear(f)
            b.launch()
            b.wait()
            before = kernel_launches()
            results = [f.collect() for f in filters[:-1]]
            assert (kernel_launches() - before > 0) == (launch == 0)
            results.append(filters[-1].collect())
            for f, (pats, text), r in zip(filters, jobs, results):
                check(f, PRM, pats, text, r)
    for f in filters:
        f.close()
