"""Timed cases of the library: what its users have it do, at their sizes.

A case is a dict of plain values. ``listed()`` names the fixed ones, ``draw``
gives others of the same kinds and ranges, ``prepare`` makes a case's inputs on
the GPU from a seed, ``run`` is one pass through the binding's calls, ``work``
the bytes that a pass cannot do without, and ``exact`` the results as plain
torch computes them in 64 bits.

Inputs and outputs are torch tensors, handed to the library as device pointers;
all cases share one context, as the calls of one program do, and no autotuner
runs, so each call takes the launch shapes that a new user gets.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opencl-sdk_gb300"))
import gbcompute as gbc  # noqa: E402

_context = None


def context():
    global _context
    if _context is None:
        _context = gbc.Context(0)
    return _context


def listed():
    return [
        # The smallest sort of key-value pairs in the library's own tests: an index or a small table sorted inside a
        # larger program, where the call's latency is what counts.
        {"name": "sort_pairs_4k", "kind": "sort", "key": "uint32", "values": True, "n": 4097, "and_words": 1,
         "descending": False},
        # Keys-only sort of 2^24 uniform 32-bit keys, the ordinary in-memory sort.
        {"name": "sort_keys_16m", "kind": "sort", "key": "uint32", "values": False, "n": 1 << 24, "and_words": 1,
         "descending": False},
        # Key-value sort of 2^28 pairs, the benchmark's default workload and the largest plain sort.
        {"name": "sort_pairs_256m", "kind": "sort", "key": "uint32", "values": True, "n": 1 << 28, "and_words": 1,
         "descending": False},
        # Device-wide exclusive scan with its exact total, the benchmark's size: offsets from counts.
        {"name": "scan_i32_1g", "kind": "scan", "dtype": "int32", "n": 1 << 30, "exclusive": True},
        # A sum of a million values read back by the host: the blocking call of an iterative program.
        {"name": "reduce_i32_1m", "kind": "reduce", "dtype": "int32", "n": 1 << 20},
        # 256-bin histogram of 2^30 bytes, the benchmark's size: an image or a byte stream.
        {"name": "histogram_u8_1g", "kind": "histogram", "dtype": "uint8", "n": 1 << 30, "bins": 256},
        # Conversion of 100 million sensor words (the reference's compute-pipeline sample) and the readings above a
        # threshold kept: transform and copy_if at an odd size.
        {"name": "filter_100m", "kind": "filter", "n": 100_000_007},
        # Batched sort and scan of 200,000 arrays of uneven length, the benchmark's batch.
        {"name": "segments_200k", "kind": "segments", "key": "uint64", "values": True, "segments": 200_000,
         "median": 256},
        # Learned-CDF sort of 2^28 floats of a mixture, the benchmark's size.
        {"name": "learned_f32_256m", "kind": "learned", "n": 1 << 28},
        # Sort, reduce by key and histogram of 2^29 Zipf-distributed 64-bit keys, the benchmark's aggregation.
        {"name": "aggregate_u64_512m", "kind": "aggregate", "n": 1 << 29, "distinct": 1 << 24},
        # Compression of timestamps and back, the benchmark's recipe at an odd size.
        {"name": "bitpack_200m", "kind": "bitpack", "n": 200_000_003, "delta": True, "step": 50},
        # A hash table of 2^26 keys filled and queried, half of the queries absent.
        {"name": "map_64m", "kind": "map", "n": 1 << 26},
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n | 1 if rng.random() < 0.7 else n

    kind = rng.choice(["sort", "sort", "sort", "scan", "reduce", "histogram", "filter", "segments", "learned", "aggregate",
                       "bitpack", "map"])
    if kind == "sort":
        return {"kind": kind, "key": rng.choice(["uint32", "int32", "float32", "uint64"]),
                "values": rng.random() < 0.5, "n": size(1 << 10, (1 << 28) - 2), "and_words": rng.choice([1, 1, 2, 4]),
                "descending": rng.random() < 0.25}
    if kind == "scan":
        return {"kind": kind, "dtype": rng.choice(["int32", "int32", "uint32", "int64"]), "n": size(1 << 10, (1 << 29) - 2),
                "exclusive": rng.random() < 0.5}
    if kind == "reduce":
        return {"kind": kind, "dtype": rng.choice(["int32", "int64"]), "n": size(1 << 10, (1 << 28) - 2)}
    if kind == "histogram":
        dtype = rng.choice(["uint8", "uint8", "uint16", "float32"])
        return {"kind": kind, "dtype": dtype, "n": size(1 << 12, (1 << 29) - 2),
                "bins": rng.choice([64, 256]) if dtype != "uint16" else rng.choice([256, 65536])}
    if kind == "filter":
        return {"kind": kind, "n": size(1 << 12, (1 << 28) - 2)}
    if kind == "segments":
        return {"kind": kind, "key": rng.choice(["uint32", "uint64", "float32"]), "values": rng.random() < 0.6,
                "segments": size(100, 200_000), "median": int(round(math.exp(rng.uniform(math.log(16), math.log(256)))))}
    if kind == "learned":
        return {"kind": kind, "n": size(1 << 21, (1 << 28) - 2)}
    if kind == "aggregate":
        return {"kind": kind, "n": size(1 << 16, (1 << 28) - 2), "distinct": size(1 << 10, 1 << 24)}
    if kind == "bitpack":
        return {"kind": kind, "n": size(1 << 12, 200_000_000), "delta": rng.random() < 0.7, "step": size(2, 1 << 16)}
    return {"kind": kind, "n": size(1 << 12, (1 << 26) - 2)}


# ---- inputs -----------------------------------------------------------------

_STORAGE = {"uint32": torch.int32, "int32": torch.int32, "float32": torch.float32, "uint64": torch.int64,
            "int64": torch.int64, "uint8": torch.uint8, "uint16": torch.int16}


def _words(n, bits, g):
    """n uniform words of 32 or 64 bits."""
    if bits == 32:
        return torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=g)
    return torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda", generator=g)


def _sort_keys(key, n, and_words, g):
    """Uniform words, or the AND of several (lower entropy); floats are normal variates."""
    if key == "float32":
        return torch.randn(n, device="cuda", generator=g) * (10.0 ** and_words)
    keys = _words(n, 64 if key == "uint64" else 32, g)
    for _ in range(and_words - 1):
        keys &= _words(n, 64 if key == "uint64" else 32, g)
    return keys


def _mixture(n, g):
    """75% from 8 Gaussians of widths over four decades, 20% lognormal, 5% copies of 1,000 values; shuffled."""
    n75, n20 = int(0.75 * n), int(0.20 * n)
    means = torch.rand(8, device="cuda", generator=g) * 2e3 - 1e3
    sigmas = torch.exp((torch.rand(8, device="cuda", generator=g) * 2 - 1) * math.log(100.0))
    which = torch.randint(0, 8, (n75,), device="cuda", generator=g)
    a = means[which] + sigmas[which] * torch.randn(n75, device="cuda", generator=g)
    b = torch.exp(2.0 * torch.randn(n20, device="cuda", generator=g))
    pool = torch.cat([a[:500], b[:500]])
    c = pool[torch.randint(0, 1000, (n - n75 - n20,), device="cuda", generator=g)]
    keys = torch.cat([a, b, c])
    del a, b, c, which
    return keys[torch.randperm(n, device="cuda", generator=g)].contiguous()


def _zipf(n, distinct, g):
    """Zipf(1.1) ranks over `distinct` values, mapped by splitmix64."""
    cdf = np.cumsum(np.arange(1, distinct + 1, dtype=np.float64) ** -1.1)  # on the host: the same sums every time
    cdf = torch.from_numpy(cdf / cdf[-1]).cuda()
    keys = torch.empty(n, dtype=torch.int64, device="cuda")
    for i in range(0, n, 1 << 26):
        u = torch.rand(min(1 << 26, n - i), device="cuda", generator=g, dtype=torch.float64)
        x = torch.searchsorted(cdf, u).clamp_(max=distinct - 1) + (-7046029254386353131)
        x = (x ^ ((x >> 30) & ((1 << 34) - 1))) * (-4658895280553007687)
        x = (x ^ ((x >> 27) & ((1 << 37) - 1))) * (-7723592293110705685)
        keys[i:i + u.numel()] = x ^ ((x >> 31) & ((1 << 33) - 1))
    return keys


def _lengths(case):
    """The batch's segment lengths (lognormal, sigma 2); a seed only changes their order."""
    lens = np.random.default_rng(case["segments"]).lognormal(math.log(case["median"]), 2.0, case["segments"])
    return np.clip(np.rint(lens), 1, 1 << 20).astype(np.int64)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ctx, kind, s = context(), case["kind"], {"case": case}
    if kind == "sort":
        n = case["n"]
        s["keys"] = _sort_keys(case["key"], n, case["and_words"], g)
        s["keys_out"] = torch.empty_like(s["keys"])
        if case["values"]:
            s["vals"] = torch.arange(n, dtype=torch.int32, device="cuda")
            s["vals_out"] = torch.empty_like(s["vals"])
    elif kind == "scan":
        s["x"] = torch.randint(0 if case["dtype"] == "uint32" else -1000, 1001, (case["n"],),
                               dtype=_STORAGE[case["dtype"]], device="cuda", generator=g)
        s["y"] = torch.empty_like(s["x"])
        s["total"] = torch.empty(1, dtype=torch.int64, device="cuda")
    elif kind == "reduce":
        s["x"] = torch.randint(-1000, 1001, (case["n"],), dtype=_STORAGE[case["dtype"]], device="cuda", generator=g)
        s["buffer"] = gbc.DeviceBuffer.wrap(ctx, s["x"].data_ptr(), case["n"], case["dtype"])
    elif kind == "histogram":
        n = case["n"]
        if case["dtype"] == "float32":
            s["x"] = torch.rand(n, device="cuda", generator=g)
        elif case["dtype"] == "uint16":
            s["x"] = torch.randint(-(1 << 15), 1 << 15, (n,), dtype=torch.int16, device="cuda", generator=g)
        else:
            s["x"] = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g)
        s["hist"] = torch.empty(case["bins"], dtype=torch.int32, device="cuda")
    elif kind == "filter":
        n = case["n"]
        s["x"] = torch.randint(0, 1000, (n,), dtype=torch.int32, device="cuda", generator=g)
        s["y"] = torch.empty(n, dtype=torch.float32, device="cuda")
        s["kept"] = torch.zeros(n, dtype=torch.float32, device="cuda")
        s["buffers"] = [gbc.DeviceBuffer.wrap(ctx, s[k].data_ptr(), n, t)
                        for k, t in (("x", np.uint32), ("y", np.float32), ("kept", np.float32))]
    elif kind == "segments":
        lens = np.random.default_rng(seed).permutation(_lengths(case))
        total = s["n"] = int(lens.sum())
        s["offsets"] = torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)).cuda()
        s["keys"] = _sort_keys(case["key"], total, 1, g)
        s["keys_out"] = torch.empty_like(s["keys"])
        if case["values"]:
            s["vals"] = torch.arange(total, dtype=torch.int32, device="cuda")
            s["vals_out"] = torch.empty_like(s["vals"])
        s["x"] = torch.randint(-1000, 1001, (total,), dtype=torch.int32, device="cuda", generator=g)
        s["y"] = torch.empty_like(s["x"])
    elif kind == "learned":
        s["keys"] = _mixture(case["n"], g)
        s["keys_out"] = torch.empty_like(s["keys"])
    elif kind == "aggregate":
        n = case["n"]
        s["keys"] = _zipf(n, case["distinct"], g)
        s["vals"] = torch.randint(0, 1 << 16, (n,), dtype=torch.int32, device="cuda", generator=g)
        s["keys_out"], s["vals_out"] = torch.empty_like(s["keys"]), torch.empty_like(s["vals"])
        s["runs"], s["sums"] = torch.zeros_like(s["keys"]), torch.zeros_like(s["keys"])
        s["counts"] = torch.zeros_like(s["vals"])
        s["hist"] = torch.empty(65536, dtype=torch.int32, device="cuda")
    elif kind == "bitpack":
        n = case["n"]
        if case["delta"]:  # slowly increasing timestamps
            steps = torch.randint(0, case["step"], (n,), dtype=torch.int64, device="cuda", generator=g)
            s["x"] = ((1_700_000_000 + torch.cumsum(steps, 0)) & 0xFFFFFFFF).to(torch.int32)
            del steps
        else:  # small values around a base
            s["x"] = torch.randint(1000, 1000 + case["step"], (n,), dtype=torch.int32, device="cuda", generator=g)
        s["capacity"] = gbc.bitpack_words_bound(n)
        s["packed"] = torch.zeros(s["capacity"], dtype=torch.int32, device="cuda")
        s["back"] = torch.empty_like(s["x"])
    elif kind == "map":
        n = case["n"]
        start = int(torch.randint(0, 1 << 30, (1,), generator=g, device="cuda"))
        numbers = torch.arange(n, dtype=torch.int64, device="cuda") + start
        s["keys"] = ((numbers * 2654435761 & 0x7FFFFFFF) * 2).to(torch.int32)  # distinct: an odd factor modulo 2^31
        del numbers
        s["vals"] = torch.randint(0, 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=g)
        s["queries"] = s["keys"][torch.randperm(n, device="cuda", generator=g)].contiguous()
        s["queries"][1::2] |= 1  # odd keys were never inserted
        s["n"], s["found"] = n, torch.empty_like(s["vals"])
        s["map"] = gbc.StaticMap(ctx, 2 * n)
    return s


# ---- one pass ---------------------------------------------------------------

def _pointer(s, name):
    return s[name].data_ptr() if name in s else 0


def run(s):
    case, ctx = s["case"], context()
    kind = case["kind"]
    if kind == "sort":
        gbc.sort_raw(ctx, s["keys"].data_ptr(), s["keys_out"].data_ptr(), case["key"], case["n"], _pointer(s, "vals"),
                     _pointer(s, "vals_out"), case["descending"])
        return [s["keys_out"], s["vals_out"]] if case["values"] else s["keys_out"]
    if kind == "scan":
        gbc.scan_raw(ctx, s["x"].data_ptr(), s["y"].data_ptr(), case["n"], case["dtype"], exclusive=case["exclusive"],
                     total_device=s["total"].data_ptr())
        return [s["y"], s["total"]]
    if kind == "reduce":
        return int(gbc.reduce(ctx, s["buffer"]))
    if kind == "histogram":
        gbc.histogram_even_raw(ctx, s["x"].data_ptr(), case["n"], case["dtype"], s["hist"].data_ptr(), case["bins"],
                               *_range(case))
        return s["hist"]
    if kind == "filter":
        x, y, kept = s["buffers"]
        gbc.transform(ctx, x, y, "x * 0.18f + 32.0f")
        count = gbc.copy_if(ctx, y, kept, "x > 100.0f")
        return [s["y"], s["kept"], count]  # kept: zeros after the first `count`
    if kind == "segments":
        gbc.segmented_sort_raw(ctx, s["keys"].data_ptr(), s["keys_out"].data_ptr(), case["key"], s["n"],
                               s["offsets"].data_ptr(), case["segments"], _pointer(s, "vals"), _pointer(s, "vals_out"))
        gbc.segmented_scan_raw(ctx, s["x"].data_ptr(), s["y"].data_ptr(), s["n"], np.int32, s["offsets"].data_ptr(),
                               case["segments"], exclusive=True)
        return [s["keys_out"], s["y"]] + ([s["vals_out"]] if case["values"] else [])
    if kind == "learned":
        gbc.sort_learned(ctx, s["keys"].data_ptr(), s["keys_out"].data_ptr(), np.float32, case["n"])
        return s["keys_out"]
    if kind == "aggregate":
        gbc.sort_raw(ctx, s["keys"].data_ptr(), s["keys_out"].data_ptr(), np.uint64, case["n"], s["vals"].data_ptr(),
                     s["vals_out"].data_ptr())
        runs = gbc.reduce_by_key_raw(ctx, s["keys_out"].data_ptr(), np.uint64, s["vals_out"].data_ptr(), case["n"],
                                     s["runs"].data_ptr(), s["sums"].data_ptr(), s["counts"].data_ptr(),
                                     s["hist"].data_ptr())
        return [s["keys_out"], s["vals_out"], s["runs"], s["sums"], s["counts"], s["hist"], runs]
    if kind == "bitpack":
        words = gbc.compress_bitpack_raw(ctx, s["x"].data_ptr(), case["n"], s["packed"].data_ptr(), s["capacity"],
                                         delta=case["delta"])
        gbc.decompress_bitpack_raw(ctx, s["packed"].data_ptr(), words, case["n"], s["back"].data_ptr(),
                                   delta=case["delta"])
        return [s["packed"], s["back"], words]
    s["map"].clear()
    added = s["map"].insert_raw(s["keys"].data_ptr(), s["vals"].data_ptr(), s["n"])
    s["map"].find_raw(s["queries"].data_ptr(), s["n"], s["found"].data_ptr())
    return [added, s["found"]]


def _range(case):
    """The histogram's [lower, upper): every value of the type, or floats in [0, 1)."""
    return {"uint8": (0.0, 256.0), "uint16": (0.0, 65536.0), "float32": (0.0, 1.0)}[case["dtype"]]


# ---- what a pass cannot do without --------------------------------------------

def work(case):
    kind = case["kind"]
    item = {k: torch.empty(0, dtype=t).element_size() for k, t in _STORAGE.items()}
    if kind == "sort":
        size = 2 * case["n"] * (item[case["key"]] + (4 if case["values"] else 0))
    elif kind == "scan":
        size = 2 * case["n"] * item[case["dtype"]]
    elif kind == "reduce":
        size = case["n"] * item[case["dtype"]]
    elif kind == "histogram":
        size = case["n"] * item[case["dtype"]] + 4 * case["bins"]
    elif kind == "filter":  # words in, floats out and in again, the readings over 100 (x > 377 of 1,000) out
        size = case["n"] * (4 + 4 + 4 + 4 * 0.622)
    elif kind == "segments":  # the sort's pairs and the scan's words, in and out
        size = 2 * int(_lengths(case).sum()) * (item[case["key"]] + 4 + 4 * case["values"])
    elif kind == "learned":
        size = 8 * case["n"]
    elif kind == "aggregate":  # pairs in and out, sorted pairs in; the runs' 20 bytes each are far fewer
        size = case["n"] * 36
    elif kind == "bitpack":  # words in, packed out and in, words out
        bits = math.log2(max(2, case["step"])) + (1 if case["delta"] else 0)
        size = case["n"] * (8 + 2 * min(32.0, math.ceil(bits)) / 8)
    else:  # pairs in, two slots per key cleared and one filled; queries, their slots and results
        size = case["n"] * (8 + 16 + 8 + 4 + 8 + 4)
    return {"bytes": size, "flops": 0}


# ---- the same results from plain torch, in 64 bits ------------------------------

def _sorted_order(keys, key, descending=False):
    """The stable order of the keys, and the keys in it."""
    ordered = keys.to(torch.float64) if key == "float32" else keys
    if key in ("uint32", "uint64"):  # signed order of the words with the top bit flipped is the unsigned one
        ordered = keys ^ (-(1 << 31) if key == "uint32" else -(1 << 63))
    order = torch.sort(ordered, stable=True, descending=descending).indices
    del ordered
    return order, keys[order]


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "sort":
        order, keys = _sorted_order(s["keys"], case["key"], case["descending"])
        keys = keys.double() if case["key"] == "float32" else keys
        return [keys, order.to(torch.int32)] if case["values"] else keys
    if kind == "scan":
        total = s["x"].sum(dtype=torch.int64)
        sums = torch.cumsum(s["x"], 0, dtype=torch.int64)
        if case["exclusive"]:
            sums -= s["x"]
        return [sums.to(s["x"].dtype), total.reshape(1)]
    if kind == "reduce":
        return int(s["x"].sum(dtype=torch.int64))
    if kind == "histogram":
        if case["dtype"] == "float32":
            bins = (s["x"].double() * case["bins"]).to(torch.int64)
        else:
            bins = (s["x"].to(torch.int64) & 0xFFFF) * case["bins"] // int(_range(case)[1])
        return torch.bincount(bins, minlength=case["bins"]).to(torch.int32)
    if kind == "filter":
        y = s["x"].double() * 0.18 + 32.0
        return [y, None, None]  # the kept readings follow the comparison of the rounded ones
    if kind == "segments":
        # a stable order by key, then a stable order of the segments' numbers in it
        lens = (s["offsets"][1:] - s["offsets"][:-1]).to(torch.int64)
        number = torch.repeat_interleave(torch.arange(case["segments"], device="cuda", dtype=torch.int32), lens)
        order, _ = _sorted_order(s["keys"], case["key"])
        order = order[torch.sort(number[order], stable=True).indices]
        keys = s["keys"][order]
        keys = keys.double() if case["key"] == "float32" else keys
        sums = torch.cumsum(s["x"], 0, dtype=torch.int64) - s["x"]
        sums = (sums - sums[s["offsets"][:-1].to(torch.int64)][number.to(torch.int64)]).to(torch.int32)
        return [keys, sums] + ([order.to(torch.int32)] if case["values"] else [])
    if kind == "learned":
        return torch.sort(s["keys"].double()).values
    if kind == "aggregate":
        order, keys = _sorted_order(s["keys"], "uint64")
        vals = s["vals"][order]
        del order
        runs, counts = torch.unique_consecutive(keys, return_counts=True)
        ends = torch.cumsum(counts, 0)
        sums = torch.cumsum(vals, 0, dtype=torch.int64)[ends - 1]
        sums[1:] -= sums[:-1].clone()
        hist = torch.bincount(keys & 0xFFFF, minlength=65536).to(torch.int32)
        for k, v in (("runs", runs), ("sums", sums), ("counts", counts)):
            s[k][:v.numel()] = v
        return [keys, vals, s["runs"], s["sums"], s["counts"], hist, runs.numel()]
    if kind == "bitpack":
        return [None, s["x"], None]
    table = torch.sort(s["keys"])
    at = torch.searchsorted(table.values, s["queries"]).clamp_(max=s["n"] - 1)
    hit = table.values[at] == s["queries"]
    return [s["n"], torch.where(hit, s["vals"][table.indices[at]], torch.full_like(s["vals"], -1))]
