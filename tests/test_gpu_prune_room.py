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
