"""The tuned scan with LEN as an argument: every word offset and byte remainder of the block that leaves the window,
both kernel forms (to 31, 33 to 63), sparse and dense modes, S = 0 (no cache-region probe) and K = 1; compared with the
oracle on texts with high bytes, newlines at every distance, and occurrences at the text's ends."""
import numpy as np
import pytest

import oracle
from ffbf_b200 import Filter, Params
from ffbf_b200 import datagen as dg

pytestmark = pytest.mark.gpu

KEYS = ("FFBF_SCAN_MODE", "FFBF_SCAN_ORDER")


def inputs(L, n, seed):
    pats = bytes(dg.gen_patterns(seed, dg.PRINTABLE, 300 if L < 8 else 2000, L, L + 25))
    text = dg.gen_text(seed + 1, dg.PRINTABLE, n, 40 if L < 30 else 120)
    rng = np.random.default_rng(seed)
    at = rng.integers(0, n, n // 500)
    text[at] = rng.integers(128, 256, at.size)
    lines = pats.split(b"\n")[:-1]
    for i, e in enumerate([L + 25, 128, 192 + L // 2, 4096 + 3, 16384, 16384 + L, n - 1, n]):
        p = np.frombuffer(lines[i % len(lines)], dtype=np.uint8)
        text[e - p.size:e] = p
    for i in range(n // 2000):
        p = np.frombuffer(lines[(7 * i) % len(lines)], dtype=np.uint8)
        text[1000 + 2000 * i:1000 + 2000 * i + p.size] = p
    return pats, text


def check(prm, pats, text):
    o = oracle.Oracle.from_params(prm)
    o.build(pats)
    s = o.scan(text)
    with Filter(prm) as f:
        f.add_patterns(pats)
        r = f.process(text)
        np.testing.assert_array_equal(r.hit_offsets, s["hits"])
        np.testing.assert_array_equal(r.line_start, s["line_start"])
        np.testing.assert_array_equal(r.line_end, s["line_end"])
        np.testing.assert_array_equal(f.get_filters()[1], o.ff)
        return s["hits"].size, f.config()[1]


@pytest.mark.parametrize("L", [1, 2, 3, 4, 5, 7, 8, 11, 12, 14, 17, 18, 21, 25, 30, 31, 33, 34, 36, 39, 40, 47, 50, 55,
                               60, 62, 63])
def test_lengths(L, monkeypatch):
    prm = Params(L, 5, 2, 1 << 19, 1 << 23)
    pats, text = inputs(L, 200_003, L)
    for env in ({}, {"FFBF_SCAN_MODE": "3"}, {"FFBF_SCAN_MODE": "1", "FFBF_SCAN_ORDER": "1"},
                {"FFBF_SCAN_MODE": "1", "FFBF_SCAN_ORDER": "2"}):
        for k in KEYS:
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        hits, mode = check(prm, pats, text)
        assert hits > 50 and ("FFBF_SCAN_MODE" not in env or mode == int(env["FFBF_SCAN_MODE"]))


@pytest.mark.parametrize("L,k,s", [(10, 1, 1), (40, 1, 1), (12, 2, 0), (20, 5, 0), (45, 4, 0), (63, 11, 0), (9, 3, 3),
                                   (33, 4, 4), (13, 2, 1), (48, 6, 3)])
def test_probe_counts(L, k, s, monkeypatch):
    prm = Params(L, k, s, 1 << 18, 1 << 21)
    pats, text = inputs(L, 300_001, 100 + L)
    for mode in (None, "0", "1"):
        for key in KEYS:
            monkeypatch.delenv(key, raising=False)
        if mode:
            monkeypatch.setenv("FFBF_SCAN_MODE", mode)
        hits, ran = check(prm, pats, text)
        assert hits > 50
        if s == 0:
            assert ran == 1, "without a cache-region probe only the dense mode applies"
        if k == 1:
            assert ran != 1, "K = 1 has no second probe"


def test_smallest_regions():
    """Cache regions of 32 and 64 bits, whose stage-1 tables are smaller than a bulk copy's granule."""
    for c in (32, 64, 128):
        prm = Params(24, 4, 2, c, 1 << 16)
        pats, text = inputs(24, 100_001, c)
        check(prm, pats[: 24 * 30], text)
