"""Results finished by one launch (up to 16384 hit windows, pruned ids or matches), at the sizes where that path can go
wrong: no hit, the edges of a CTA's share (128 and 1024 windows), the most it takes and one more, windows crowded into
a small part of the text, lines that reach over more tiles than it walks, several pattern ids per offset, and batch jobs
with more windows than their room. Everything equals the oracle."""
import numpy as np
import pytest

import oracle
from ffbf_b200 import Batch, Filter, Params
from ffbf_b200 import datagen as dg

pytestmark = pytest.mark.gpu

PRM = Params(20, 5, 2, 1 << 22, 1 << 26)


def planted(n_hits, nbytes, seed, newline=80, span=None, dup=1):
    """Patterns (each written `dup` times to the file) and a text with n_hits occurrences of them, no two overlapping,
    within the first `span` bytes; the lines the occurrences sit in keep their '\\n'."""
    pats = dg.gen_patterns(seed, dg.PRINTABLE, 500, 20, 30)
    lines = bytes(pats).split(b"\n")[:-1]
    text = dg.gen_text(seed + 1, dg.PRINTABLE, nbytes, newline)
    span = span or nbytes
    step = span // max(n_hits, 1)
    assert n_hits == 0 or step >= 31
    for i in range(n_hits):
        p = lines[i % len(lines)]
        at = i * step + (i * 7) % (step - 30)
        text[at:at + len(p)] = np.frombuffer(p, dtype=np.uint8)
    return bytes(pats) * dup, text


def check(f, prm, pats, text, r):
    o = oracle.Oracle.from_params(prm)
    o.build(pats)
    s = o.scan(text)
    pr = o.prune(pats)
    off, pid = o.verify(pats, pr["ids"], text, s["hits"])
    np.testing.assert_array_equal(r.hit_offsets, s["hits"])
    np.testing.assert_array_equal(r.line_start, s["line_start"])
    np.testing.assert_array_equal(r.line_end, s["line_end"])
    np.testing.assert_array_equal(f.filter_phrases(), pr["ids"])
    m = f.verify()
    np.testing.assert_array_equal(m[0], off)
    np.testing.assert_array_equal(m[1], pid)
    return s["hits"].size


@pytest.mark.parametrize("n_hits", [0, 1, 127, 128, 129, 1024, 1025, 16383, 16384, 16385])
def test_result_sizes(n_hits):
    pats, text = planted(n_hits, 2_000_003, 11 + n_hits)
    with Filter(PRM) as f:
        f.add_patterns(pats)
        assert check(f, PRM, pats, text, f.process(text)) >= n_hits


@pytest.mark.parametrize("n_hits,nbytes,newline,span,dup", [
    (3000, 32 << 20, 80, 100_000, 1),       # crowded: one bucket of the sort would hold them all
    (300, 3 << 20, 3_000_000, None, 1),     # about one '\n': lines reach over all tiles
    (2000, 1 << 20, 80, None, 5),           # five pattern ids per offset
    (4000, 1 << 20, 80, None, 5),           # 20000 matches of 4000 windows
])
def test_uneven_results(n_hits, nbytes, newline, span, dup):
    pats, text = planted(n_hits, nbytes, 3 * n_hits, newline, span, dup)
    with Filter(PRM) as f:
        f.add_patterns(pats)
        assert check(f, PRM, pats, text, f.process(text)) >= n_hits


def test_batch_results_within_and_over_their_room():
    """A batch collects each job's windows into room for one per 8 KiB of text (at least 512); jobs with more are
    collected alone. Results hold over repeated launches and after the batch is gone."""
    import torch

    jobs = [planted(n, b, 900 + n) for n, b in ((0, 5000), (511, 300_000), (512, 300_001), (513, 300_002),
                                               (2000, 1 << 20), (20, 40 << 20))]
    filters, texts = [], []
    b = Batch()
    for pats, text in jobs:
        filters.append(Filter(PRM))
        filters[-1].add_patterns(pats)
        texts.append(torch.from_numpy(text).cuda())
        b.add(filters[-1], texts[-1].data_ptr(), text.size)
    b.prepare()
    b.wait()  # nothing launched yet: nothing to collect
    for _ in range(2):
        b.launch()
        b.wait()
    b.wait()
    b.close()
    for f, (pats, text) in zip(filters, jobs):
        check(f, PRM, pats, text, f.collect())
        f.close()
