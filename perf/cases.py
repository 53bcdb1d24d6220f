"""Timed cases: what programs have this matcher do, each through the calls such a program makes.

Every case names its filter geometry (LEN, K, S, log2 of the cache and external regions' bits), its pattern set
(count and lengths of `alphabet`: 0 printable, 1 lowercase words, 2 bytes) and its text. Kinds:

  lines   strings tested one at a time against a resident filter (operator[])
  resident  a host text scanned with a resident filter, then the feed-forward prune and the exact matches
  device  the same for a text that already is in device memory
  cli     one run of the command with a filter cache: a new filter, patterns, the cache's image, one host
          text, and the bytes of every file the command writes
  full    a large pinned host text against a resident filter: scan, candidate lines, prune, exact matches
  build   a new filter from a pattern file, and the cache image the command would save
  batch   many (filter, device text) jobs prepared once and launched together
  serve   a burst of requests to a scan server over its resident sets
"""
import numpy as np
import torch

from ffbf_b200 import Batch, Filter, Params, Server
from ffbf_b200 import datagen as dg

KiB, MiB, GiB = 1 << 10, 1 << 20, 1 << 30

PLAIN = dict(len=20, k=5, s=2, cache_log2=24, ext_log2=28, alphabet=0, len_lo=20, len_hi=40, newline=80)
WORDS = dict(len=32, k=5, s=2, cache_log2=23, ext_log2=26, alphabet=1, len_lo=32, len_hi=64, newline=100)
BYTES = dict(len=16, k=5, s=2, cache_log2=24, ext_log2=28, alphabet=2, len_lo=16, len_hi=16, newline=0)
DEFAULT = dict(len=19, k=5, s=2, cache_log2=24, ext_log2=28, alphabet=0, len_lo=19, len_hi=50, newline=80)


def listed():
    return [
        # an editor or a log filter asking about single lines: calls per second count
        dict(DEFAULT, name="lines", kind="lines", patterns=10_000, text=24_001, plants=60),
        # one small document against a resident pattern set: latency counts
        dict(PLAIN, name="document_100k", kind="resident", patterns=10_000, text=100_003, plants=5),
        # `ffbf patterns out < corpus` where the pattern file's filter cache exists
        dict(DEFAULT, name="cli_8m", kind="cli", patterns=50_000, text=8 * MiB + 4_321, plants=400),
        # an ordinary text on the device, few patterns
        dict(PLAIN, name="plain_64m", kind="device", patterns=10_000, text=64 * MiB, plants=500),
        # a large text, few patterns, a ragged end
        dict(PLAIN, name="plain_1g", kind="device", patterns=10_000, text=GiB + 12_345, plants=8_000),
        # the largest text: a million patterns over 4 GiB of words
        dict(WORDS, name="words_4g", kind="device", patterns=1_000_000, text=4 * GiB, plants=20_000),
        # virus-style signatures over raw bytes
        dict(BYTES, name="signatures_2g", kind="device", patterns=4_000_000, text=2 * GiB + 777, plants=25_000),
        # long patterns with a geometry of the user's own
        dict(len=40, k=6, s=2, cache_log2=23, ext_log2=27, alphabet=0, len_lo=40, len_hi=80, newline=120,
             name="long_256m", kind="device", patterns=150_000, text=256 * MiB + 99, plants=2_000),
        # many customers' texts, each with its own pattern set
        dict(name="batch_48", kind="batch", jobs=48, patterns=64_000, text=32 * MiB, plants=0),
        # a scan service: a burst of uneven requests over resident sets
        dict(WORDS, name="serve_64", kind="serve", sets=4, requests=64, patterns=150_000, text=48 * MiB, plants=200),
        # a new pattern file: build its filter and write the cache
        dict(WORDS, name="build_1m", kind="build", patterns=1_000_000, text=0, plants=0),
        # a corpus read from disk into pinned memory, everything the command prints wanted
        dict(WORDS, name="full_512m", kind="full", patterns=1_000_000, text=512 * MiB + 1, plants=2_500),
    ]


def _log_uniform(rng, lo, hi):
    return int(lo * (hi / lo) ** rng.random())


def _geometry(rng, patterns):
    """A tuned or another LEN, and regions that suit the pattern count."""
    if rng.random() < 0.6:
        g = dict(rng.choice([PLAIN, WORDS, DEFAULT]))
    else:
        n = rng.choice([16, 24, 24, rng.randint(8, 63), rng.randint(8, 63)])
        k = rng.choice([5, 5, 4, 6, 7])
        g = dict(len=n, k=k, s=rng.choice([1, 2, 2, 2, 3]), alphabet=rng.choice([0, 0, 1]) if n >= 24 else 0, len_lo=n,
                 len_hi=n + rng.randint(0, 40), newline=rng.choice([60, 80, 100, 200]))
        c = 20 if patterns < 16_000 else 22 if patterns < 64_000 else 23
        g.update(cache_log2=c, ext_log2=c + 4)
    return g


def draw(rng):
    kind = rng.choice(["lines", "resident", "resident", "cli", "device", "device", "device", "device", "full", "build",
                       "batch", "serve"])
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(8, 48), patterns=_log_uniform(rng, 4_000, 64_000),
                    text=_log_uniform(rng, MiB, 32 * MiB), plants=0)
    if kind == "device" and rng.random() < 0.2:
        n = _log_uniform(rng, 32 * MiB, 2 * GiB)
        return dict(BYTES, kind=kind, patterns=_log_uniform(rng, 10_000, 4_000_000), text=n,
                    plants=max(1, n // 80_000))
    patterns = _log_uniform(rng, 1_000, 1_000_000)
    g = _geometry(rng, patterns)
    if kind == "serve":
        return dict(g, kind=kind, sets=rng.randint(2, 5), requests=rng.randint(8, 64),
                    patterns=min(patterns, 200_000), text=_log_uniform(rng, 8 * MiB, 48 * MiB), plants=200)
    lo, hi = {"lines": (24_000, 96_000), "resident": (20_000, 24 * MiB), "cli": (MiB, 24 * MiB),
              "device": (MiB, 2 * GiB), "full": (32 * MiB, 512 * MiB), "build": (1, 1)}[kind]
    n = _log_uniform(rng, lo, hi) if kind != "build" else 0
    plants = 0 if kind == "build" else n // 400 if kind == "lines" else max(4, n // 150_000)
    return dict(g, kind=kind, patterns=patterns, text=n, plants=plants)


def _params(c):
    return Params(c["len"], c["k"], c["s"], 1 << c["cache_log2"], 1 << c["ext_log2"])


def _table(c):
    """65536 bytes whose uniform draws have the case's letter and line-length distribution."""
    if c["alphabet"] == 1:
        w = np.array([1.0 / (i + 1) for i in range(26)])
        p = np.concatenate([[1 / 7], w / w.sum() * 6 / 7])
        symbols = np.concatenate([[0x20], np.arange(26) + 0x61])
    else:
        p = np.full(95, 1 / 95)
        symbols = np.arange(95) + 0x20
    n_nl = 65536 // c["newline"]
    edges = np.floor(np.cumsum(p) * (65536 - n_nl) + 0.5).astype(np.int64)
    t = np.full(65536, 10, dtype=np.uint8)
    at = 0
    for s, e in zip(symbols, edges):
        t[at:e] = s
        at = e
    return torch.from_numpy(t).cuda()


def _device_text(c, seed, n, patterns, plants):
    """n bytes of the case's text on the device, with `plants` pattern occurrences at stratified offsets."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    table = None if c["alphabet"] == 2 else _table(c)
    for a in range(0, n, 256 * MiB):
        m = min(256 * MiB, n - a)
        if table is None:
            out[a:a + m] = torch.randint(0, 256, (m,), dtype=torch.uint8, device="cuda", generator=g)
        else:
            i = torch.randint(0, 65536, (m,), dtype=torch.int32, device="cuda", generator=g)
            torch.index_select(table, 0, i, out=out[a:a + m])
            del i
    ends = np.flatnonzero(patterns == 10)
    starts = np.concatenate([[0], ends[:-1] + 1])
    plants = min(plants, n // (c["len_hi"] + 1))
    if plants:
        rng = np.random.default_rng(seed)
        ids = rng.integers(0, starts.size, plants)
        lens = (ends - starts)[ids]
        stride = n // plants
        offs = np.arange(plants) * stride + (rng.random(plants) * (stride - c["len_hi"])).astype(np.int64)
        within = np.arange(lens.sum()) - np.repeat(np.cumsum(lens) - lens, lens)
        to = torch.from_numpy(np.repeat(offs, lens) + within).cuda()
        out[to] = torch.from_numpy(patterns[np.repeat(starts[ids], lens) + within]).cuda()
    return out


def _patterns(c, seed):
    return dg.gen_patterns(seed, c["alphabet"], c["patterns"], c["len_lo"], c["len_hi"])


def _filter(c, patterns):
    f = Filter(_params(c))
    f.add_patterns(patterns)
    return f


def _pinned(t):
    h = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _batch_jobs(c, seed):
    """The batched workload's jobs within the case's limits (dg.batched: sizes and counts log-uniform)."""
    jobs = dg.batched(c["jobs"], 1_000, c["patterns"], 256 * KiB, c["text"], seed=seed)
    return [dict(len=w.params.len, k=w.params.k, s=w.params.s, alphabet=0, newline=80, len_lo=w.len_lo, len_hi=w.len_hi,
                 cache_log2=w.params.cache_bits.bit_length() - 1, ext_log2=w.params.ext_bits.bit_length() - 1,
                 patterns=w.n_patterns, text=w.text_bytes, plants=w.n_plant, seed=w.seed % (1 << 62)) for w in jobs]


class _Results:
    """The program's own result buffers, of one size for all seeds: every array is kept there, whole, with its
    length in "n"; what a shorter result leaves of the one before is cleared."""

    def __init__(self, c):
        jobs = _batch_jobs(c, 0) if c["kind"] == "batch" else [c] * c.get("sets", 1)
        hits = 4_096.0
        for j in jobs:  # planted windows and the filter's expected false positives
            fill_c = 1 - np.exp(-j["s"] * j["patterns"] / 2.0 ** j["cache_log2"])
            fill_e = 1 - np.exp(-(j["k"] - j["s"]) * j["patterns"] / 2.0 ** j["ext_log2"])
            hits += 16 * (j["plants"] + j["text"] * fill_c ** j["s"] * fill_e ** (j["k"] - j["s"]))
        self.cap = int(hits) * (4 if len(jobs) > 1 else 1)
        self.line = 2 * c.get("newline", 100)
        self.pattern_bytes = c["patterns"] * (c.get("len_hi", 0) + 9)
        self.image_bytes = 4 * c.get("k", 0) * c["patterns"]
        self.bufs = {}

    def keep(self, **arrays):
        out = {"n": np.array([a.size for a in arrays.values()])}
        for name, a in arrays.items():
            if name not in self.bufs:
                cap = {"stdout": self.cap * self.line // 4, "image": self.image_bytes, "pruned": self.pattern_bytes,
                       "index": self.pattern_bytes}.get(name, self.cap)
                self.bufs[name] = [np.zeros(cap, dtype=a.dtype), 0]
            buf, used = self.bufs[name]
            n = min(a.size, buf.size)
            buf[:n] = a[:n]
            buf[n:used] = 0
            self.bufs[name][1] = n
            out[name] = buf
        return out


def prepare(c, seed):
    kind = c["kind"]
    s = {"kind": kind, "out": _Results(c)}
    if kind == "batch":
        s["batch"], s["filters"], s["texts"] = Batch(), [], []
        for j in _batch_jobs(c, seed):
            pats = _patterns(j, j["seed"])
            f = _filter(j, pats)
            t = _device_text(j, j["seed"], j["text"], pats, j["plants"])
            s["filters"].append(f)
            s["texts"].append(t)
            torch.cuda.synchronize()
            s["batch"].add(f, t.data_ptr(), t.numel())
        s["batch"].prepare()
        return s
    if kind == "serve":
        s["server"], pool = Server(), []
        for i in range(c["sets"]):
            pats = _patterns(c, seed * 16 + i)
            s["server"].add_set(_filter(c, pats))
            pool.append(_device_text(c, seed * 16 + i, c["text"] // c["sets"], pats, c["plants"]))
        s["pool"] = _pinned(torch.cat(pool))
        rng = np.random.default_rng(seed)
        sizes = np.minimum(np.exp(np.log(MiB) + 1.5 * rng.standard_normal(c["requests"])), s["pool"].size).astype(int)
        sizes = np.maximum(sizes, 1)
        s["requests"] = [(int(rng.integers(c["sets"])), int(rng.integers(s["pool"].size - n + 1)), int(n))
                         for n in sizes]
        return s
    pats = _patterns(c, seed)
    s["params"], s["patterns"] = _params(c), pats
    if kind == "build":
        return s
    text = _device_text(c, seed, c["text"], pats, c["plants"])
    if kind == "device":
        s["text"] = text
    elif kind == "full":
        s["text"] = _pinned(text)
    else:
        s["text"] = text.cpu().numpy()
    if kind == "lines":
        s["lines"] = [x for x in s["text"].tobytes().split(b"\n") if x][:48]
        s["lines"].append(s["text"].tobytes()[: c["text"] // 4].replace(b"\n", b" "))  # and one long one
    if kind == "cli":
        with _filter(c, pats) as f:
            s["image"] = f.save_filter()
    else:
        s["filter"] = _filter(c, pats)
    torch.cuda.synchronize()
    return s


def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def _results(f, scan):
    ids = f.filter_phrases()
    offsets, pids = f.verify()
    return dict(hits=scan.hit_offsets, line_start=scan.line_start, line_end=scan.line_end, ids=ids,
                match_offsets=offsets, match_ids=pids)


def run(s):
    kind, out = s["kind"], s["out"]
    if kind == "lines":
        return np.array([s["filter"].test_line(x) for x in s["lines"]])
    if kind == "resident":
        s["filter"].clear_ff()
        return out.keep(**_results(s["filter"], s["filter"].process(s["text"])))
    if kind == "device":
        s["filter"].clear_ff()
        s["filter"].process_device(s["text"].data_ptr(), s["text"].numel())
        return out.keep(**_results(s["filter"], s["filter"].collect()))
    if kind == "cli":
        with Filter(s["params"]) as f:
            f.set_patterns(s["patterns"])
            f.load_filter(s["image"])
            f.process(s["text"])
            lines = f.format_lines(s["text"])
            f.filter_phrases()
            pruned, index = f.format_pruned()
        return out.keep(stdout=_bytes(lines), pruned=_bytes(pruned), index=_bytes(index))
    if kind == "full":
        f = s["filter"]
        f.clear_ff()
        scan = f.process(s["text"])
        lines = f.format_lines(s["text"])
        return out.keep(stdout=_bytes(lines), **_results(f, scan))
    if kind == "build":
        with Filter(s["params"]) as f:
            f.add_patterns(s["patterns"])
            return out.keep(image=_bytes(f.save_filter()))
    if kind == "batch":
        s["batch"].launch()
        s["batch"].wait()
        got = [f.collect() for f in s["filters"]]
    else:
        server = s["server"]
        order = {server.submit(si, s["pool"][o:o + n]): i for i, (si, o, n) in enumerate(s["requests"])}
        got = [None] * len(order)
        left = len(order)
        while left:
            for r in server.poll(wait_us=2000):
                got[order[r.request_id]] = r
                left -= 1
    kept = out.keep(**{k: np.concatenate([getattr(r, k) for r in got])
                       for k in ("hit_offsets", "line_start", "line_end")})
    kept["per_text"] = np.array([r.hit_offsets.size for r in got])
    return kept


def work(c):
    """Each text byte and pattern byte read once; a new filter's bits written once (its image for a build)."""
    if c["kind"] == "batch":  # the mean of the jobs' log-uniform text sizes
        lo, hi = 256 * KiB, c["text"]
        n = c["jobs"] * (hi - lo) / np.log(hi / lo) if hi > lo else c["jobs"] * lo
        return {"bytes": float(n), "flops": 0.0}
    if c["kind"] == "serve":
        return {"bytes": float(c["requests"] * min(3.08 * MiB, c["text"])), "flops": 0.0}
    pattern_bytes = c["patterns"] * ((c["len_lo"] + c["len_hi"]) / 2 + 1)
    n = float(c["text"])
    if c["kind"] == "build":
        n += pattern_bytes + 4.0 * c["k"] * c["patterns"]
    if c["kind"] == "cli":
        n += pattern_bytes + 4.0 * c["k"] * c["patterns"] + ((1 << c["cache_log2"]) + (1 << c["ext_log2"])) / 8
    return {"bytes": n, "flops": 0.0}
