"""The tuned scan at the edges of its streams, tiles and work items: texts that end on and around a row, a stream, a
16 KiB tile and a CTA's streams, with occurrences that end on the last byte and straddle the last whole stream's end, in
the sparse mode and each dense probe order, and texts whose only '\\n' lies after the last whole stream. Windows, lines and
the feed-forward filter equal the oracle's."""
import numpy as np
import pytest

import oracle
from ffbf_b200 import Filter, Params
from ffbf_b200 import datagen as dg

pytestmark = pytest.mark.gpu

KEYS = ("FFBF_SCAN_MODE", "FFBF_SCAN_ORDER", "FFBF_SCAN_THREADS")
VARIANTS = [{"FFBF_SCAN_MODE": "3"}, {"FFBF_SCAN_MODE": "0", "FFBF_SCAN_THREADS": "384"},
            {"FFBF_SCAN_MODE": "1", "FFBF_SCAN_ORDER": "0"}, {"FFBF_SCAN_MODE": "1", "FFBF_SCAN_ORDER": "1"},
            {"FFBF_SCAN_MODE": "1", "FFBF_SCAN_ORDER": "2"}]
SIZES = [16384, 16385, 16384 + 127, 16384 + 128, 16384 + 129, 32768 - 1, 100_003, 192 * 128, 192 * 128 + 1,
         512 * 128 * 5 - 1, 2_500_001, 9_000_077]


@pytest.fixture
def scan_env(monkeypatch):
    def use(env):
        for k in KEYS:
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
    return use


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
    return s


@pytest.mark.parametrize("L", [16, 20, 32])
def test_ends_of_streams_and_texts(L, scan_env):
    prm = Params(L, 5, 2, 1 << 18, 1 << 22)
    pats = bytes(dg.gen_patterns(L, dg.PRINTABLE, 3000, L, L + 20))
    lines = [np.frombuffer(x, dtype=np.uint8) for x in pats.split(b"\n")[:-1]]
    for n in SIZES:
        text = dg.gen_text(n, dg.PRINTABLE, n, 300)
        # occurrences at the text's end, across every row boundary near it, and across some inner ones
        ends = [n] + [n // 128 * 128 - 128 * k + d for k in range(18) for d in (L // 2,)] + \
               [128 * k + 7 for k in range(3, n // 128, max(1, n // 128 // 50))]
        for i, e in enumerate(ends):
            p = lines[i % len(lines)]
            if L <= len(p) <= e <= n:
                text[e - len(p):e] = p
        for env in VARIANTS:
            scan_env(env)
            s = check(prm, pats, text)
            assert s["hits"].size and s["hits"][-1] + L <= n
    scan_env({})


@pytest.mark.parametrize("n", [16384 + 100, 40_000, 2_500_001])
def test_newlines_only_at_the_end(n, scan_env):
    prm = Params(20, 5, 2, 1 << 18, 1 << 22)
    pats = bytes(dg.gen_patterns(5, dg.PRINTABLE, 500, 20, 40))
    base = dg.gen_text(n, dg.PRINTABLE, n, 0)
    base[base == 10] = ord("x")
    dg.plant(6, np.frombuffer(pats, dtype=np.uint8), base, 20)
    for at in ([], [n - 1], [n // 128 * 128], [n // 128 * 128 - 1, n - 2]):
        text = base.copy()
        for a in at:
            text[min(a, n - 1)] = 10
        for env in VARIANTS[:1] + VARIANTS[3:4]:
            scan_env(env)
            check(prm, pats, text)
    scan_env({})
