"""The pruned pattern file and its index for small and large files, few and many surviving lines, with and without a final
newline, asked for twice: the oracle's bytes, however the lines come back from the device."""
import numpy as np
import pytest

import oracle
from ffbf_b200 import Filter, Params
from ffbf_b200 import datagen as dg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("newline", [True, False])
@pytest.mark.parametrize("n,keep", [(300, 1), (300, 300), (20_000, 40), (20_000, 4_999), (20_000, 5_001), (20_000, 20_000)])
def test_pruned_files(n, keep, newline):
    prm = Params(20, 5, 2, 1 << 22, 1 << 26)
    pats = dg.gen_patterns(n + keep, dg.PRINTABLE, n, 20, 60)
    ends = np.flatnonzero(pats == 10)
    text = b"".join(bytes(pats[ends[i - 1] + 1 if i else 0:ends[i] + 1]) for i in range(n - keep, n))
    pats = bytes(pats) if newline else bytes(pats)[:-1]
    text = np.frombuffer(text, dtype=np.uint8)
    o = oracle.Oracle.from_params(prm)
    o.build(pats)
    o.scan(text)
    want = o.prune(pats)
    assert want["ids"].size >= keep
    with Filter(prm) as f:
        f.add_patterns(pats)
        f.process(text)
        np.testing.assert_array_equal(f.filter_phrases(), want["ids"])
        for _ in range(2):
            out, index = f.format_pruned()
            assert out == want["out"] and index == want["index"]
        # other patterns: nothing of the old file is left
        other = dg.gen_patterns(3, dg.PRINTABLE, 50, 20, 30)
        f.add_patterns(other)
        f.process(other)
        o.build(other)
        o.scan(other)
        f.filter_phrases()
        assert f.format_pruned()[0] == o.prune(other)["out"]
