"""The prune when its first id buffer does not fit the HBM budget: it emits the ids a second time, and the pinned room
that both passes write is the caller's again when the call returns."""
import numpy as np
import pytest

from ffbf_b200 import FFBFError, Filter, Params
from ffbf_b200 import datagen as dg

pytestmark = pytest.mark.gpu


def test_second_emission_is_waited_for():
    pats = dg.gen_patterns(5, dg.PRINTABLE, 32_000_000, 16, 16)  # an emission of some 200 microseconds
    text = pats[:17 * 1000]
    with Filter(Params(16, 5, 2, 1 << 27, 1 << 28)) as f:
        f.add_patterns(pats)
        f.process(text)
        # the smallest budget that suffices leaves less than the 16384 ids that the first buffer would hold
        for budget in range(1 << 30, 1 << 31, 48 << 10):
            f.set_hbm_budget(budget)
            try:
                ids = f.filter_phrases()
                break
            except FFBFError as e:
                assert e.status == 2, e
        hit = f.test_line(b"\x01" * 3000)
        assert not hit
        assert 1000 <= ids.size <= 6144
        f.set_hbm_budget(0)
        np.testing.assert_array_equal(ids, f.filter_phrases())


@pytest.mark.parametrize("n", [8192 * 1024, 8192 * 1024 + 1, 8193 * 1024 + 5, 2 * 16384 * 1024 - 3])
def test_ids_around_the_block_prefix(n):
    """Pattern sets of 8192 blocks of 1024, where the emission still sums the counts itself, and more."""
    pats = dg.gen_patterns(7, dg.PRINTABLE, n, 16, 16)
    lines = pats.reshape(n, 17)
    keep = np.unique(np.concatenate([np.arange(0, n, 9973), [1023, 1024, n - 1025, n - 2, n - 1]]))
    with Filter(Params(16, 5, 2, 1 << 28, 1 << 30)) as f:
        f.add_patterns(pats)
        f.process(lines[keep].reshape(-1).copy())
        ids = f.filter_phrases()
        f.verify()
    # a survivor that was not in the text is a false positive of the feed-forward filter, or another copy of a line
    assert np.isin(keep, ids).all()
    assert (np.diff(ids.astype(np.int64)) > 0).all() and ids[-1] == n - 1
    assert ids.size <= keep.size + 8
