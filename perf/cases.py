"""The work that a program has this framework do, as cases that can be timed.

``listed()`` holds the named cases, ``draw(rng)`` gives one more of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call (a
matcher over its pattern set, new input bytes, output buffers), ``run(state)``
is one scan through the public entry points, and ``work(case)`` the bytes it
cannot do without.

Every kind of scan returns its whole match set.  The host-facing entry points
return it sorted; the device-resident ones append matches in no particular
order, so ``run`` brings them into the canonical order on the device, as a
program that reports them does: a match becomes one 64-bit key and the keys are
sorted (places past the match count hold the largest key).
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import warpstate_b200 as ws

KIB, MIB, GIB = 1 << 10, 1 << 20, 1 << 30
PRINTABLE = bytes(range(0x20, 0x7F))
LOWER = b"abcdefghijklmnopqrstuvwxyz"
LOG_ALPHABET = LOWER + b"ABCDEFGHIJ0123456789_=:.- \n"
JOINS = ["[0-9]", "[A-F]", "[G-M]", "[N-T]", "[U-Z]", "[_.-]", "[ ]", "[0-4]", "[5-9]"]
IUPAC = {"R": "AG", "Y": "CT", "S": "CG", "W": "AT", "K": "GT", "M": "AC",
         "B": "CGT", "D": "AGT", "H": "ACT", "V": "ACG", "N": "ACGT"}
LAST = (1 << 63) - 1


def listed():
    return [
        # one short record (a packet, a log line group) against a mixed rule
        # set, host bytes in and matches out: latency is all there is
        {"name": "host_4k", "kind": "host", "bytes": 4 * KIB, "literals": 100, "regexes": 20},
        # one document or file, an odd length, the same rules
        {"name": "host_1m", "kind": "host", "bytes": 1000003, "literals": 100, "regexes": 20},
        # a log followed in 1 MiB reads through the stream pipeline, exact across reads
        {"name": "stream_24m", "kind": "stream", "bytes": 24 * MIB + 77, "piece": MIB, "literals": 100, "regexes": 20},
        # a small literal set over a buffer that fits the L2 cache
        {"name": "literals_16m", "kind": "literals", "bytes": 16 * MIB, "literals": 100, "fold": False,
         "shortest": 4, "longest": 16},
        # a large signature set over a large buffer
        {"name": "literals_1g", "kind": "literals", "bytes": GIB, "literals": 10000, "fold": False,
         "shortest": 8, "longest": 32},
        # keyword search that ignores case, with short keywords, ragged length
        {"name": "literals_nocase_96m", "kind": "literals", "bytes": 96 * MIB + 1234567, "literals": 1000, "fold": True,
         "shortest": 3, "longest": 20},
        # a rule set of 500 regexes as the default configuration lays it out
        # (several automata), a mid-sized buffer
        {"name": "regex_64m", "kind": "regex", "bytes": 64 * MIB, "regexes": 500, "states": 0, "chunk": 0},
        # the layout the autotuner picks for such sets (one automaton, 8 KiB
        # chunks), a large buffer
        {"name": "regex_1g", "kind": "regex", "bytes": GIB, "regexes": 160, "states": 32768, "chunk": 8192},
        # log rules with line anchors and word boundaries
        {"name": "anchored_32m", "kind": "anchored", "bytes": 32 * MIB + 4099, "regexes": 40},
        # rules with unbounded repeats (numbers, identifiers, blanks of any length)
        {"name": "unbounded_200m", "kind": "unbounded", "bytes": 200 * MIB + 13, "regexes": 60},
        # many small documents in one call, literals and regexes together
        {"name": "batch_40k", "kind": "batch", "items": 40000, "literals": 1500, "regexes": 200},
        # a genome-sized nucleotide input, k-mers and degenerate motifs, 64-bit offsets
        {"name": "dna_2g", "kind": "dna", "bytes": 2 * GIB, "literals": 20000, "regexes": 100},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm, odd ones among them."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["host", "stream", "literals", "regex", "anchored", "unbounded", "batch", "dna"])
    if kind == "host":
        return {"kind": kind, "bytes": _log(rng, 200, 4 * MIB), "literals": _log(rng, 10, 1000),
                "regexes": rng.randint(1, 60)}
    if kind == "stream":
        return {"kind": kind, "bytes": _log(rng, MIB, 48 * MIB), "piece": _log(rng, 128 * KIB, 8 * MIB),
                "literals": _log(rng, 10, 1000), "regexes": rng.randint(1, 60)}
    if kind == "literals":
        size, count = _log(rng, MIB, GIB), _log(rng, 20, 10000)
        # three-letter words come in small sets (each occurs everywhere)
        shortest = rng.choice([3, 4, 5, 6, 8, 12] if count <= 1000 and size <= 128 * MIB else [4, 5, 6, 8, 12])
        return {"kind": kind, "bytes": size, "literals": count, "fold": rng.random() < 0.3, "shortest": shortest,
                "longest": shortest + rng.randint(4, 24)}
    if kind == "regex":
        return {"kind": kind, "bytes": _log(rng, 256 * KIB, GIB), "regexes": _log(rng, 5, 150),
                "states": rng.choice([0, 0, 32768]), "chunk": rng.choice([0, 0, 8192])}
    if kind == "anchored":
        return {"kind": kind, "bytes": _log(rng, 256 * KIB, 64 * MIB), "regexes": rng.randint(4, 60)}
    if kind == "unbounded":
        return {"kind": kind, "bytes": _log(rng, 256 * KIB, 256 * MIB), "regexes": rng.randint(4, 80)}
    if kind == "batch":
        return {"kind": kind, "items": _log(rng, 100, 40000), "literals": _log(rng, 20, 1500),
                "regexes": rng.randint(5, 120)}
    return {"kind": kind, "bytes": _log(rng, 16 * MIB, 2 * GIB), "literals": _log(rng, 500, 20000),
            "regexes": rng.randint(10, 100)}


# --------------------------------------------------------------- pattern sets
def _word(r, alphabet, lo, hi, weights=None):
    return bytes(r.choices(alphabet, weights=weights, k=r.randint(lo, hi)))


def _alternation(words):
    return "(?:" + "|".join(w.decode() for w in words) + ")"


def _members(cls):
    """The characters of one of the classes of JOINS."""
    body, out, i = cls[1:-1], [], 0
    while i < len(body):
        if i + 2 < len(body) and body[i + 1] == "-":
            out += [chr(c) for c in range(ord(body[i]), ord(body[i + 2]) + 1)]
            i += 3
        else:
            out.append(body[i])
            i += 1
    return out


def _literals(n, alphabet, lo, hi, seed):
    """n distinct literals; character frequencies fall off as text's do."""
    r = random.Random(seed)
    letters = list(alphabet)
    r.shuffle(letters)
    weights = [1.0 / (k + 2) ** 0.8 for k in range(len(letters))]
    out = {}
    while len(out) < n:
        out[_word(r, letters, lo, hi, weights)] = True
    return list(out)


def _joined_regexes(n, seed):
    """Two alternations of words joined by a short class run, and a matching text each."""
    r = random.Random(seed)
    out = []
    for _ in range(n):
        a = [_word(r, b"abcdefghijklmnop", 4, 12) for _ in range(r.randint(2, 4))]
        b = [_word(r, b"abcdefghijklmnop", 4, 12) for _ in range(r.randint(2, 4))]
        cls = r.choice(JOINS)
        mid = "".join(r.choices(_members(cls), k=r.randint(1, 8)))
        out.append((_alternation(a) + cls + "{1,8}" + _alternation(b), r.choice(a) + mid.encode() + r.choice(b)))
    return out


def _anchored_regexes(n, seed):
    """Log rules: line starts and ends, word boundaries."""
    r = random.Random(seed)
    out = []
    for k in range(n):
        w = [_word(r, LOWER, 4, 9) for _ in range(3)]
        d = str(r.randint(100, 999)).encode()
        out.append([
            (r"\b" + _alternation(w) + r"\b", b" " + w[0] + b" "),
            (r"^" + w[0].decode() + "[=:][0-9]{1,6}", b"\n" + w[0] + b":" + d),
            (w[1].decode() + r" [a-z]{2,8}\.?$", w[1] + b" " + w[2][:6] + b"\n"),
            (r"\b" + w[2].decode() + r"=[A-J]{1,4}[0-9]{2}\b", b" " + w[2] + b"=BAD42 "),
        ][k % 4])
    return out


def _unbounded_regexes(n, seed):
    """Rules with repeats of any length; every fourth one is bounded."""
    r = random.Random(seed)
    out = []
    for k in range(n):
        w = [_word(r, LOWER, 4, 8) for _ in range(3)]
        d = str(r.randint(1, 10 ** 9)).encode()
        out.append([
            (w[0].decode() + "=[0-9]+", w[0] + b"=" + d),
            (_alternation(w[:2]) + "[ :]+[0-9_]+" + "[.]", w[1] + b":  " + d + b"."),
            (w[2].decode() + "_[a-z0-9_]*[A-J]", w[2] + b"_" + d + b"ab_cD"),
            (_alternation(w) + "[-:][A-J]{1,3}", w[0] + b"-CAB"),
        ][k % 4])
    return out


def _iupac_regexes(n, seed):
    r = random.Random(seed)
    codes = sorted(IUPAC)
    out = []
    for _ in range(n):
        pos = [r.choice("ACGT") if r.random() < 0.85 else r.choice(codes) for _ in range(r.randint(20, 40))]
        out.append(("".join(c if c in "ACGT" else "[" + IUPAC[c] + "]" for c in pos),
                    "".join(r.choice(IUPAC.get(c, c)) for c in pos).encode()))
    return out


def _patterns(case):
    """(literals, regexes with a matching text each) of a case's rule set."""
    kind, n = case["kind"], case.get("literals", 0)
    if kind in ("host", "stream"):
        return _literals(n, LOWER, 5, 16, 101), _joined_regexes(case["regexes"], 102)
    if kind == "literals":
        alphabet = LOWER if case["literals"] <= 200 else PRINTABLE
        return _literals(n, alphabet, case["shortest"], case["longest"], 103), []
    if kind == "regex":
        return [], _joined_regexes(case["regexes"], 104)
    if kind == "anchored":
        return [], _anchored_regexes(case["regexes"], 105)
    if kind == "unbounded":
        return [], _unbounded_regexes(case["regexes"], 106)
    if kind == "batch":
        return _literals(n, PRINTABLE, 6, 24, 107), _joined_regexes(case["regexes"], 108)
    return _literals(n, b"ACGT", 20, 32, 109), _iupac_regexes(case["regexes"], 110)


@functools.lru_cache(maxsize=None)
def _matcher(key):
    """The matcher that a program builds once for its rule set and keeps, texts
    that its patterns match, and how many literals a byte of text starts by
    chance."""
    case = dict(key)
    literals, regexes = _patterns(case)
    builder = ws.PatternSet.builder()
    for p in literals:
        builder = builder.literal_bytes(p)
    for source, _ in regexes:
        builder = builder.regex(source)
    if case.get("fold"):
        builder = builder.case_insensitive(True)
    config = ws.AutoMatcherConfig()
    states = case.get("states") or (32768 if case["kind"] == "dna" else 0)
    chunk = case.get("chunk") or (8192 if case["kind"] == "dna" else 0)
    if states:
        config = config.dfa_max_states(states)
    if chunk:
        config = config.walk_chunk(chunk)
    letters = 26 if case.get("literals", 0) <= 200 else 40
    chance = sum(float(letters) ** -len(p) for p in literals)
    matcher = ws.GpuMatcher.with_config(builder.build(), config)
    return matcher, literals[:2048] + [text for _, text in regexes], chance


def _matcher_of(case):
    return _matcher(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "bytes", "items", "piece"))))


# --------------------------------------------------------------------- inputs
def _markov(n, alphabet, gen, dev, blank=None):
    """n bytes of order-1 Markov text over `alphabet` (one fixed language per
    alphabet), many chains side by side."""
    r = np.random.default_rng(len(alphabet))
    k = len(alphabet)
    table = np.empty((k, 256), dtype=np.int64)
    for s in range(k):
        w = 1.0 / (r.permutation(k) + 2.0) ** 0.7
        for c, p in (blank or {}).items():
            w[alphabet.index(c)] = p * w.sum()
        cut = np.round(np.cumsum(w / w.sum()) * 256).astype(np.int64)
        table[s] = np.searchsorted(cut, np.arange(256), side="right").clip(0, k - 1)
    following = torch.from_numpy(table * 256).to(dev).reshape(-1)
    letters = torch.tensor(list(alphabet), dtype=torch.uint8, device=dev)
    steps = min(2048, max(64, n // 1024))
    out = torch.empty(n, dtype=torch.uint8, device=dev)
    for at in range(0, n, 512 * MIB):
        m = min(512 * MIB, n - at)
        chains = -(-m // steps)
        draws = torch.randint(0, 256, (steps, chains), dtype=torch.uint8, device=dev, generator=gen)
        state = torch.randint(0, k, (chains,), dtype=torch.int64, device=dev, generator=gen) * 256
        text = torch.empty((steps, chains), dtype=torch.uint8, device=dev)
        for i in range(steps):
            state = following.take(state + draws[i])
            text[i] = state >> 8
        flat = text.t().reshape(-1)[:m]
        out[at:at + m] = letters.take(flat.long()) if m < 64 * MIB else _spell(flat, letters)
        del draws, text, flat
    return out


def _spell(codes, letters):
    """letters[codes], in slices (the index of a lookup is 64-bit)."""
    out = torch.empty_like(codes)
    for at in range(0, codes.numel(), 64 * MIB):
        part = codes[at:at + 64 * MIB]
        out[at:at + part.numel()] = letters.take(part.long())
    return out


def _uniform(n, alphabet, gen, dev):
    letters = torch.tensor(list(alphabet), dtype=torch.uint8, device=dev)
    return _spell(torch.randint(0, len(alphabet), (n,), dtype=torch.uint8, device=dev, generator=gen), letters)


def _overwrite(data, texts, places, which, dev):
    """Writes texts[which[i]] at places[i]."""
    longest = max(len(t) for t in texts)
    rows = np.zeros((len(texts), longest), dtype=np.uint8)
    for i, t in enumerate(texts):
        rows[i, :len(t)] = np.frombuffer(t, dtype=np.uint8)
    rows = torch.from_numpy(rows).to(dev)
    lens = torch.tensor([len(t) for t in texts], device=dev)
    cols = torch.arange(longest, device=dev)
    inside = cols[None, :] < lens[which][:, None]
    at = places[:, None] + cols[None, :]
    data[at[inside]] = rows[which][inside]


def _plant(data, texts, slot, gen, dev):
    """One matching text in each slot, at a place of its own."""
    longest = max(len(t) for t in texts)
    slot = max(slot, 2 * longest)
    n = data.numel() // slot
    if not n:
        return
    places = torch.arange(n, device=dev) * slot
    places += torch.randint(0, slot - longest, (n,), device=dev, generator=gen)
    _overwrite(data, texts, places, torch.randint(0, len(texts), (n,), device=dev, generator=gen), dev)


def _nucleotides(n, gen, dev):
    """Uniform ACGT, about 1% of it in runs of N."""
    data = _uniform(n, b"ACGT", gen, dev)
    runs = [b"N" * k for k in range(1, 51)]
    count = int(n * 0.01 / 25.5)
    places = torch.randint(0, n - 50, (count,), device=dev, generator=gen)
    for at in range(0, count, 1 << 18):
        part = places[at:at + (1 << 18)]
        _overwrite(data, runs, part, torch.randint(0, 50, (part.numel(),), device=dev, generator=gen), dev)
    return data


def _item_sizes(n, seed):
    """Document sizes: lognormal, median 4 KiB, 64 B to 1 MiB (the same total for every seed's order)."""
    r = np.random.default_rng(7 * n)
    sizes = np.clip(np.exp(np.log(4096) + 1.5 * r.standard_normal(n)), 64, MIB - 1).astype(np.int64)
    return np.random.default_rng(seed).permutation(sizes)


def _total(case):
    return int(_item_sizes(case["items"], 0).sum()) if case["kind"] == "batch" else case["bytes"]


def _slot(case):
    """Bytes per planted match."""
    if case["kind"] in ("literals", "regex", "anchored", "unbounded"):
        return 16 * KIB if case["bytes"] > 256 * MIB else 64 * KIB if case["bytes"] > 4 * MIB else 4 * KIB
    return {"host": 4 * KIB, "stream": 16 * KIB, "batch": 16 * KIB, "dna": MIB}[case["kind"]]


def _input(case, seed, texts, dev):
    kind, n = case["kind"], _total(case)
    gen = torch.Generator(device=dev).manual_seed(seed)
    if kind == "dna":
        data = _nucleotides(n, gen, dev)
    elif kind == "literals" and case["literals"] <= 200:
        data = _uniform(n, LOWER, gen, dev)
    elif kind in ("host", "stream", "anchored", "unbounded"):
        data = _markov(n, LOG_ALPHABET, gen, dev, blank={0x20: 0.14, 0x0A: 0.012})
    else:
        data = _markov(n, PRINTABLE, gen, dev)
    _plant(data, texts, min(_slot(case), max(256, n // 8)), gen, dev)
    return data


def prepare(case, seed):
    matcher, texts, chance = _matcher_of(case)
    dev, kind, n = "cuda:0", case["kind"], _total(case)
    data = _input(case, seed, texts, dev)
    # room for half as many matches again as are expected
    cap = 1 << int(1.5 * (n // _slot(case) + n // (4 * MIB) + n * chance + 256)).bit_length()
    if kind == "host":
        return {"kind": kind, "matcher": matcher, "data": data.cpu().numpy().tobytes(),
                "table": np.zeros((cap, 3), dtype=np.int64)}
    if kind == "stream":
        return {"kind": kind, "pipeline": ws.StreamPipeline.new(matcher), "data": data.cpu().numpy(),
                "piece": case["piece"], "table": np.zeros((cap, 3), dtype=np.int64)}
    state = {"kind": kind, "matcher": matcher, "data": data, "bytes": n, "cap": cap,
             "count": torch.zeros(1, dtype=torch.int64, device=dev), "place": torch.arange(cap, device=dev),
             "last": torch.full((1,), LAST, device=dev)}
    if kind == "batch":  # ws_tagged_match: source_id (64-bit), pattern_id, start, end, reserved
        sizes = _item_sizes(case["items"], seed)
        state["ends"] = torch.from_numpy(np.cumsum(sizes).astype(np.uint32).view(np.int32)).to(dev)
        state["ids"] = torch.arange(case["items"], dtype=torch.int64, device=dev)
        state["out"] = torch.zeros((cap, 6), dtype=torch.int32, device=dev)
        # id, start (20 bits), pattern (12 bits), length (8 bits)
        state["weights"] = torch.tensor([1 << 40, 0, 1 << 8, (1 << 20) - 1, 1, 0], device=dev)
    elif kind == "dna":  # ws_match64: pattern_id, reserved, start, end (64-bit)
        state["out"] = torch.zeros((cap, 6), dtype=torch.int32, device=dev)
        # start (31 bits), pattern (16 bits), length (16 bits)
        state["weights"] = torch.tensor([1 << 16, 0, (1 << 32) - 1, 0, 1, 0], device=dev)
    else:  # ws_match: pattern_id, start, end
        state["out"] = torch.zeros((cap, 3), dtype=torch.int32, device=dev)
        state["weights"] = torch.tensor([1 << 16, (1 << 32) - 1, 1], device=dev)
    return state


def run(state):
    kind = state["kind"]
    if kind in ("host", "stream"):  # the rows go into the program's own table
        if kind == "host":
            rows = state["matcher"].scan_array(state["data"])
        else:
            rows = state["pipeline"].scan_array(state["data"], block=state["piece"])
        state["table"][:len(rows)] = rows
        state["table"][len(rows):] = 0
        return {"count": len(rows), "matches": state["table"]}
    m, stream = state["matcher"], torch.cuda.current_stream().cuda_stream
    data, out, count = state["data"].data_ptr(), state["out"].data_ptr(), state["count"].data_ptr()
    if kind == "batch":
        m.scan_batch_device(data, state["bytes"], state["ends"].data_ptr(), state["ids"].data_ptr(),
                            state["ids"].numel(), out, state["cap"], count, stream)
    elif kind == "dna":
        m.scan_device64(data, state["bytes"], out, state["cap"], count, stream)
    else:
        m.scan_device(data, state["bytes"], out, state["cap"], count, stream)
    keys = (state["out"] * state["weights"]).sum(1)
    keys = torch.where(state["place"] < state["count"], keys, state["last"]).sort().values
    return {"count": state["count"], "matches": keys}


def work(case):
    """The input read once; the match rows written once (one per planted text)."""
    n = _total(case)
    row = {"batch": 24, "dna": 24, "stream": 24}.get(case["kind"], 12)
    table = 12 * case["items"] if case["kind"] == "batch" else 0
    return {"bytes": n + table + row * (n // _slot(case)), "flops": 0}
