"""operator[] over lines around the kernel's block of 256 windows and around the pinned room that short lines are read
from, with the only hit in the first or the last window."""
import numpy as np
import pytest

from ffbf_b200 import Filter, Params
from ffbf_b200 import datagen as dg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 19, 63])
def test_hit_in_first_and_last_window(L):
    prm = Params(L, 5, 2, 1 << 16, 1 << 20)
    pats = bytes(dg.gen_patterns(3, dg.PRINTABLE, 1 if L == 1 else 200, L, L))
    pat = pats.split(b"\n")[0]
    filler = b"\x01"
    with Filter(prm) as f:
        f.add_patterns(pats)
        assert not f.test_line(filler * 3000), "the filler must not hit by itself"
        for n in (L, L + 1, 255 + L - 1, 256 + L - 1, 257 + L - 1, 512 + L, 49152 - 1, 49152, 49153, 1_000_003):
            assert f.test_line(pat + filler * (n - L)), n
            assert f.test_line(filler * (n - L) + pat), n
            assert not f.test_line(filler * n), n
        assert not f.test_line(pat[:-1]) and not f.test_line(b"")
        # the scan's results are not disturbed by a test in between
        text = np.frombuffer((filler * 100 + pat + b"\n") * 400, dtype=np.uint8).copy()
        r = f.process(text)
        f.test_line(pat)
        assert r.hit_offsets.size >= 400 and f.filter_phrases().size >= 1
