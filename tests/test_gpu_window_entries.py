"""The sparse scan that keeps a window's S-box entries in registers (the compiled lengths but 32) and the one that reads
them again (32): every CTA size that launch_config takes, over texts with high bytes and newlines, against the oracle."""
import numpy as np
import pytest

import oracle
from ffbf_b200 import Filter, Params
from ffbf_b200 import datagen as dg

pytestmark = pytest.mark.gpu

MiB = 1 << 20


@pytest.mark.parametrize("cache_log2", [17, 20, 22])  # tables below 2^20 bits, of 2^20, and folded to 2^20
@pytest.mark.parametrize("L", [16, 19, 20, 24, 32])
@pytest.mark.parametrize("n", [16_384 + 77, 4 * MiB + 128, 5 * MiB + 31, 9 * MiB + 1, 17 * MiB + 12_345])
def test_sparse_scan(n, L, cache_log2, monkeypatch):
    monkeypatch.setenv("FFBF_SCAN_MODE", "3")
    prm = Params(L, 5, 2, 1 << cache_log2, 1 << (cache_log2 + 4))
    pats = bytes(dg.gen_patterns(L, dg.PRINTABLE, 1000, L, L + 25))
    text = dg.gen_text(n % 1000, dg.PRINTABLE, n, 90)
    rng = np.random.default_rng(L)
    at = rng.integers(0, n, n // 400)
    text[at] = rng.integers(128, 256, at.size)
    lines = pats.split(b"\n")[:-1]
    for i in range(40):
        p = np.frombuffer(lines[i], dtype=np.uint8)
        o = 0 if i == 0 else n - p.size if i == 1 else int(rng.integers(0, n - p.size))
        text[o:o + p.size] = p
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
        assert s["hits"].size >= 30 and f.config()[1] == 3
