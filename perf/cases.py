"""The sorts that users of this library run, as timed cases.

Every case is one call (or the two calls a program makes in a row) of the
public Python entry points on inputs of the shapes that the repository's own
benchmark and tests use: URL lists with long shared prefixes, duplicate-heavy
words, uniform strings, batches of independent instances, request streams,
delimited texts and suffixes.  Inputs are made on the GPU from a seed.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "string-sorting_b200"))
import pyssort  # noqa: E402

CHUNK = 1 << 22  # strings generated at a time
ALPHABETS = pyssort.BATCH_ALPHABETS
MAX_LENS = pyssort.BATCH_MAX_LENS
URL_MEAN, WORD_MEAN = 53.75, 8.1  # mean bytes per string, its NUL included


def listed():
    return [
        # A single short list: latency of one call.
        {"name": "words_500", "path": "device", "data": "words", "n": 500, "vocab": 1_000,
         "off": 8, "lcp": True},
        # A page-sized list of URLs, 4-byte offsets.
        {"name": "urls_20k", "path": "device", "data": "urls", "n": 20_011, "hosts": 256,
         "off": 4, "lcp": True},
        # The million uniform strings of the benchmark's plain configuration.
        {"name": "uniform_1m", "path": "device", "data": "uniform", "n": 1_000_000, "alphabet": 1,
         "max_len": 20, "off": 8, "lcp": True},
        # Order only (no LCP array asked for), a ragged size.
        {"name": "urls_3m_perm", "path": "device", "data": "urls", "n": 2_999_999, "hosts": 4096,
         "off": 4, "lcp": False},
        # The benchmark's headline: 50 M URLs with perm and LCP.
        {"name": "urls_50m", "path": "device", "data": "urls", "n": 50_000_000, "hosts": 4096,
         "off": 8, "lcp": True},
        # The duplicate-heavy configuration: 100 M copies of Zipf words.
        {"name": "words_100m", "path": "device", "data": "words", "n": 100_000_000,
         "vocab": 1_000_000, "off": 8, "lcp": True},
        # Many small independent lists in one call.
        {"name": "batch_small", "path": "batch", "instances": 200, "lo": 100, "hi": 5_000,
         "list_seed": 11, "limit": 1_000_000_000, "off": 4, "lcp": True},
        # The batched configuration: counts in [100, 2 M], 1.5e9 key bytes.
        {"name": "batch_c4", "path": "batch", "instances": 20_000, "lo": 100, "hi": 2_000_000,
         "list_seed": 5, "limit": 1_500_000_000, "off": 8, "lcp": True},
        # All suffixes of a text with copied passages (deep shared prefixes).
        {"name": "suffixes_16m", "path": "suffixes", "n": 16_000_000, "off": 4, "lcp": True},
        # A NUL-delimited text resident on the GPU: string starts, then the sort.
        {"name": "text_urls_5m", "path": "text", "n": 5_000_011, "hosts": 4096, "off": 4,
         "lcp": True},
        # A list in pinned host memory, through the copying entry point.
        {"name": "host_urls_500k", "path": "host", "n": 500_000, "hosts": 4096, "off": 8,
         "lcp": True},
        # A burst of device-resident requests of mixed sizes at the request server.
        {"name": "serve_24", "path": "serve", "requests": 24, "lo": 1_000, "hi": 2_000_000,
         "list_seed": 7, "off": 4, "lcp": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    path = rng.choice(["device"] * 6 + ["batch", "batch", "suffixes", "text", "host", "serve"])
    case = {"path": path, "off": rng.choice([4, 8]), "lcp": rng.random() < 0.8}
    if path == "device":
        case["data"] = rng.choice(["urls", "words", "uniform"])
        if case["data"] == "urls":
            case.update(n=_log(rng, 300, 50_000_000), hosts=rng.choice([64, 1024, 4096]))
        elif case["data"] == "words":
            n = _log(rng, 300, 90_000_000)
            case.update(n=n, vocab=max(200, min(1_000_000, n // rng.choice([2, 10, 50]))))
        else:
            case.update(n=_log(rng, 300, 40_000_000), alphabet=rng.randrange(3),
                        max_len=rng.choice([8, 20, 32, 128]))
            if case["max_len"] == 128:  # 64 bytes per string: keep the arena URL-sized
                case["n"] = min(case["n"], 20_000_001)
    elif path == "batch":
        hi = _log(rng, 1_000, 1_000_000)
        case.update(instances=_log(rng, 8, 400), lo=100, hi=hi, list_seed=rng.randrange(1 << 20),
                    limit=1_000_000_000)
    elif path == "suffixes":
        case.update(n=_log(rng, 50_000, 16_000_000))
    elif path == "text":
        case.update(n=_log(rng, 3_000, 20_000_000), hosts=rng.choice([64, 4096]))
    elif path == "host":
        case.update(n=_log(rng, 1_000, 2_000_000), hosts=rng.choice([64, 4096]))
    else:
        case.update(requests=rng.randrange(4, 25), lo=1_000, hi=_log(rng, 10_000, 2_000_000),
                    list_seed=rng.randrange(1 << 20))
    return case


# ---- inputs ------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(n, g):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _zipf(n, size, s, g):
    w = torch.arange(1, size + 1, device="cuda", dtype=torch.float64).pow_(-s)
    cdf = torch.cumsum(w, 0)
    return torch.searchsorted(cdf, _rand(n, g) * cdf[-1]).clamp_(max=size - 1)


def _starts(lens):
    """Start of each string when every string takes lens + 1 bytes, and the total."""
    ends = torch.cumsum(lens + 1, 0)
    return ends - (lens + 1), int(ends[-1])


def _pack(parts):
    """One arena (16 zero bytes at its end) and the int64 offsets of parts = [(bytes, starts)]."""
    total = sum(int(b.numel()) for b, _ in parts)
    arena = torch.zeros(total + 16, dtype=torch.uint8, device="cuda")
    offs, at = [], 0
    for b, s in parts:
        arena[at:at + b.numel()] = b
        offs.append(s + at)
        at += b.numel()
    return arena, torch.cat(offs)


def _uniform_part(lens, lo, size, g):
    """Strings of the given lengths, bytes uniform over size[i] values from lo[i]."""
    starts, total = _starts(lens)
    ids = torch.repeat_interleave(torch.arange(lens.numel(), device="cuda"), lens + 1,
                                  output_size=total)
    r = torch.rand(total, generator=g, device="cuda")
    b = (lo[ids] + (r * size[ids]).to(torch.int64).clamp_(max=94)).to(torch.uint8)
    b[starts + lens] = 0
    return b, starts


def _instances(counts, max_lens, alphabets, g):
    """Strings of consecutive instances: length U[1, max_len], bytes of the alphabet."""
    dev = dict(device="cuda", dtype=torch.int64)
    c = torch.tensor(counts, **dev)
    per = [torch.repeat_interleave(torch.tensor(v, **dev), c) for v in
           (max_lens, [ALPHABETS[a][0] for a in alphabets], [ALPHABETS[a][1] for a in alphabets])]
    parts = []
    for at in range(0, int(per[0].numel()), CHUNK):
        m, lo, size = (p[at:at + CHUNK] for p in per)
        lens = 1 + (_rand(m.numel(), g) * m).to(torch.int64)
        parts.append(_uniform_part(lens, lo, size, g))
    return _pack(parts)


def _urls(n, n_hosts, g):
    """"http://" + a Zipf(1.1) host of 8-24 letters + 1-6 segments "/" + 3-12 of [a-z0-9]."""
    hosts = torch.randint(97, 123, (n_hosts, 24), generator=g, device="cuda", dtype=torch.uint8)
    host_len = torch.randint(8, 25, (n_hosts,), generator=g, device="cuda")
    alnum = torch.tensor(list(b"abcdefghijklmnopqrstuvwxyz0123456789"), dtype=torch.uint8,
                         device="cuda")
    pfx = torch.tensor(list(b"http://"), dtype=torch.uint8, device="cuda")
    parts = []
    for at in range(0, n, CHUNK):
        m = min(CHUNK, n - at)
        h = _zipf(m, n_hosts, 1.1, g)
        hl = host_len[h]
        segs = torch.randint(1, 7, (m, 1), generator=g, device="cuda")
        seg = torch.randint(4, 14, (m, 6), generator=g, device="cuda")  # with its '/'
        seg *= torch.arange(6, device="cuda") < segs
        ends = torch.cumsum(seg, 1)
        lens = 7 + hl + ends[:, -1]
        starts, total = _starts(lens)
        b = alnum[torch.randint(0, 36, (total,), generator=g, device="cuda")]
        for k in range(7):
            b[starts + k] = pfx[k]
        for k in range(24):
            on = hl > k
            b[(starts + 7 + k)[on]] = hosts[h[on], k]
        for k in range(6):
            on = seg[:, k] > 0
            b[(starts + 7 + hl + ends[:, k] - seg[:, k])[on]] = 47
        b[starts + lens] = 0
        parts.append((b, starts))
    return _pack(parts)


def _words(n, vocab, g):
    """Copies of Zipf(1.0)-drawn words of a vocabulary of distinct words with
    geometric(0.15) lengths clipped to [1, 24]."""
    m = 2 * vocab + 4096
    lens = (torch.log1p(-_rand(m, g)) / math.log(0.85)).to(torch.int64).clamp_(0, 23) + 1
    chars = torch.randint(97, 123, (m, 24), generator=g, device="cuda")
    chars *= torch.arange(24, device="cuda") < lens[:, None]
    h = torch.zeros(m, dtype=torch.int64, device="cuda")
    for k in range(24):  # distinct words by a 64-bit hash of the letters
        h = h * 6364136223846793005 + chars[:, k] + 1442695040888963407
        h ^= h >> 29
    _, inv = torch.unique(h, return_inverse=True)
    first = torch.full((int(inv.max()) + 1,), m, dtype=torch.int64, device="cuda")
    first.scatter_reduce_(0, inv, torch.arange(m, device="cuda"), "amin")
    pick = torch.sort(first).values[:vocab]
    lens, chars = lens[pick], chars[pick].to(torch.uint8)
    parts = []
    for at in range(0, n, CHUNK):
        w = _zipf(min(CHUNK, n - at), int(pick.numel()), 1.0, g)
        wl = lens[w]
        starts, total = _starts(wl)
        b = torch.zeros(total, dtype=torch.uint8, device="cuda")
        for k in range(24):
            on = wl > k
            b[(starts + k)[on]] = chars[w[on], k]
        parts.append((b, starts))
    return _pack(parts)


def _repeat_text(n, seed, g):
    """Words joined by spaces, with passages of log-uniform length in [32, 4096]
    copied from one position to another, one per 80,000 bytes as in the
    benchmark's suffix text (followed by 16 zero bytes)."""
    arena, _ = _words(n // 7 + 64, min(1_000_000, max(200, n // 50)), g)
    text = torch.zeros(n + 16, dtype=torch.uint8, device="cuda")
    m = min(n, arena.numel() - 16)
    text[:m] = arena[:m]
    text[:n][text[:n] == 0] = 32
    rng = np.random.default_rng(seed)
    for _ in range(max(4, n // 80_000)):
        k = min(int(math.exp(rng.uniform(math.log(32), math.log(4096)))), n // 2)
        a, b = (int(v) for v in rng.integers(0, n - k, size=2))
        text[b:b + k] = text[a:a + k].clone()
    return text


def _offsets(offs, width):
    return offs if width == 8 else offs.to(torch.int32)


def _instance_list(case):
    """(counts, length bounds, alphabets) of a batch or a request burst."""
    rng = random.Random(case["list_seed"])
    counts, lens, alph, total = [], [], [], 0.0
    for _ in range(case.get("instances", case.get("requests", 0))):
        counts.append(int(round(math.exp(rng.uniform(math.log(case["lo"]),
                                                     math.log(case["hi"]))))))
        lens.append(rng.choice(MAX_LENS))
        alph.append(rng.randrange(3))
        total += counts[-1] * ((1 + lens[-1]) / 2 + 1)
        if total >= case.get("limit", math.inf):
            break
    return counts, lens, alph


def _strings(case, g):
    if case.get("data") == "words":
        return _words(case["n"], case["vocab"], g)
    if case.get("data") == "uniform":
        return _instances([case["n"]], [case["max_len"]], [case["alphabet"]], g)
    return _urls(case["n"], case["hosts"], g)


def _outputs(n, lcp):
    return (torch.empty(n, dtype=torch.int32, device="cuda"),
            torch.empty(n, dtype=torch.int32, device="cuda") if lcp else None)


def prepare(case, seed):
    g, path, off = _gen(seed), case["path"], case["off"]
    if path == "serve":
        counts, lens, alph = _instance_list(case)
        reqs, need, strings = [], 0, 0
        for c, m, a in zip(counts, lens, alph):
            arena, offs = _instances([c], [m], [a], g)
            reqs.append((arena, _offsets(offs, off)) + _outputs(c, case["lcp"]))
            need += arena.numel() + 512
            strings += c
        torch.cuda.synchronize()
        return {"path": path, "srv": pyssort.Server(need, strings), "reqs": reqs, "off": off}
    st = {"path": path, "off": off, "sorter": pyssort.Sorter(0)}
    if path == "batch":
        counts, lens, alph = _instance_list(case)
        arena, offs = _instances(counts, lens, alph, g)
        st["inst"] = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int64,
                                  device="cuda").to(torch.int32)
        st["ninst"] = len(counts)
    elif path == "suffixes":
        arena, offs = _repeat_text(case["n"], seed, g), None
    else:
        arena, offs = _strings(case, g)
    n = int(offs.numel()) if offs is not None else case["n"]
    st["n"], st["arena"] = n, arena
    if path == "host":
        st["arena"] = arena.cpu().pin_memory()
        st["offs"] = _offsets(offs, off).cpu().pin_memory()
        st["perm"] = torch.empty(n, dtype=torch.int32).pin_memory()
        st["lcp"] = torch.empty(n, dtype=torch.int32).pin_memory() if case["lcp"] else None
        wide = np.uint64 if off == 8 else np.uint32
        st["np"] = (st["arena"].numpy(), st["offs"].numpy().view(wide),
                    st["perm"].numpy().view(np.uint32),
                    st["lcp"].numpy().view(np.uint32) if case["lcp"] else None)
        return st
    if path in ("text", "suffixes"):  # the call below writes the string starts
        st["offs"] = torch.empty(n, dtype=torch.int32 if off == 4 else torch.int64, device="cuda")
    else:
        st["offs"] = _offsets(offs, off)
    st["perm"], st["lcp"] = _outputs(n, case["lcp"])
    torch.cuda.synchronize()
    return st


def run(st):
    path = st["path"]
    if path == "serve":
        srv = st["srv"]
        for arena, offs, perm, lcp in st["reqs"]:
            srv.submit_ptr(arena, arena.numel(), offs, st["off"], perm.numel(), perm, lcp)
        srv.drain()
        return [(perm, lcp) for _, _, perm, lcp in st["reqs"]]
    s, n = st["sorter"], st["n"]
    if path == "host":
        arena, offs, perm, lcp = st["np"]
        return s.sort_host(arena, offs, with_lcp=lcp is not None, perm=perm, lcp=lcp)
    arena, offs, perm, lcp = st["arena"], st["offs"], st["perm"], st["lcp"]
    if path == "batch":
        s.sort_batch_device(arena, arena.numel(), offs, st["off"], n, st["inst"], st["ninst"],
                            perm, lcp)
        return perm, lcp
    if path in ("text", "suffixes"):
        mode = pyssort.TEXT_RAW if path == "text" else pyssort.TEXT_SUFFIXES
        n = s.text_offsets_device(arena, arena.numel() - 16, mode, offs, st["off"], n)
    s.sort_device(arena, arena.numel(), offs, st["off"], n, perm, lcp)
    return perm, lcp


def work(case):
    if case["path"] in ("batch", "serve"):
        counts, lens, _ = _instance_list(case)
        n = sum(counts)
        text = sum(c * ((1 + m) / 2 + 1) for c, m in zip(counts, lens))
    else:
        n = case["n"]
        text = n * (1 if case["path"] == "suffixes" else
                    WORD_MEAN if case.get("data") == "words" else
                    (1 + case["max_len"]) / 2 + 1 if case.get("data") == "uniform" else URL_MEAN)
    return {"bytes": text + n * (case["off"] + 4 + (4 if case["lcp"] else 0)), "flops": 0}
