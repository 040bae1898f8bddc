"""The work whose speed this repository looks after: what its users call, at the sizes they call it with.

A case names one public entry point (or the chain of entry points that one
user-level step consists of), a seeded input of the generators of the package
and the sizes.  ``listed()`` are fixed cases, ``draw()`` makes more of the same
ranges.  Every pass goes through the Python mirror of the C ABI with its
default options and the library's default knobs; outputs are compared whole.

Every output is a whole number or a byte, so ``exact()`` has no value to add.
"""
import math

import torch

from __graft_entry__ import load_package

d = load_package()
_ctx = []


def _context():
    """The process's context: a user's program makes one per host thread and keeps it for all its calls."""
    if not _ctx:
        _ctx.append(d.Context(0))
    return _ctx[0]


def listed():
    return [
        # The smallest sort requests a server or a library call meets: launches, read-backs and latency are all there is.
        {"name": "request_1k", "kind": "request", "n": 1000, "p": 8, "min_len": 8, "max_len": 256},
        # An ordinary request of the serving mix (its sizes are log-uniform in 1e3 .. 4e6), an odd size.
        {"name": "request_60k", "kind": "request", "n": 60013, "p": 8, "min_len": 8, "max_len": 256},
        # The largest request of the serving mix.
        {"name": "request_4m", "kind": "request", "n": 4000000, "p": 8, "min_len": 8, "max_len": 256},
        # The headline workload: 32e6 strings of 200 bytes, D/N 0.25, 64 PEs.
        {"name": "dn_32m", "kind": "dn", "n": 32000000, "len": 200, "k": 50, "p": 64},
        # The largest configuration: 1e8 strings of 100 bytes, D/N 0.5.
        {"name": "dn_100m", "kind": "dn", "n": 100000000, "len": 100, "k": 50, "p": 64},
        # Skewed lengths and long common prefixes: a fifth of the strings 500 bytes long with 394 shared bytes.
        {"name": "skew_20m", "kind": "skew", "n": 20000000, "len": 100, "k": 20, "long_len": 500, "long_k": 400,
         "frac_long": 0.2, "p": 64},
        # Many suffix sets of uneven size in one batched call (deep repeats, a four-letter alphabet).
        {"name": "suffix_batch", "kind": "suffix", "nsets": 16, "lo": 1 << 14, "hi": 4 << 20, "max_len": 256, "p": 64},
        # Host buffers in and out: the end-to-end call, copies included.
        {"name": "host_1m", "kind": "host", "n": 1000003, "p": 8, "min_len": 8, "max_len": 256},
        # The merge-sort path: whole strings and LCPs per receiving PE.
        {"name": "ms_8m", "kind": "ms", "n": 8000000, "len": 200, "k": 50, "p": 64},
        # hQuicksort, the competitor of the reference's evaluation, on 16 PEs.
        {"name": "hq_6m", "kind": "hq", "n": 6000011, "len": 120, "k": 40, "p": 16},
        # The stage entries one after the other, as the reference's policy classes call them: local sort, distinguishing
        # prefixes, partition, bucket scatter, merge.
        {"name": "stages_4m", "kind": "stages", "n": 4000000, "len": 200, "k": 50, "p": 16},
        # The wire formats of the exchange between GPUs, there and back: LCPs as varints, sorted hashes Golomb-coded.
        {"name": "wire_16m", "kind": "wire", "n": 16000000, "ranges": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["request", "request", "request", "dn", "dn", "skew", "suffix", "host", "ms", "hq", "stages", "wire"])
    if kind in ("request", "host"):
        n = _log(rng, 1000, 4000000 if kind == "request" else 1000000)
        return {"kind": kind, "n": n, "p": rng.choice([2, 4, 7, 8, 16]), "min_len": 8,
                "max_len": rng.choice([64, 100, 256, 333])}
    if kind == "skew":
        n = _log(rng, 200000, 20000000)
        return {"kind": kind, "n": n, "len": rng.randint(60, 120), "k": rng.randint(12, 40),
                "long_len": rng.randint(420, 520), "long_k": rng.randint(200, 400),
                "frac_long": round(rng.uniform(0.05, 0.2), 3), "p": rng.choice([16, 31, 64])}
    if kind == "suffix":
        return {"kind": kind, "nsets": rng.randint(1, 16), "lo": 1 << 14, "hi": _log(rng, 1 << 17, 4 << 20),
                "max_len": rng.choice([128, 200, 256]), "p": rng.choice([16, 31, 64])}
    if kind == "wire":
        return {"kind": kind, "n": _log(rng, 100000, 16000000), "ranges": rng.choice([8, 31, 64])}
    length = rng.randint(50, 250)
    k = max(12, int(length * rng.uniform(0.1, 1.0)))
    if kind == "dn":
        return {"kind": kind, "n": _log(rng, 100000, min(100000000, 6400000000 // (length + 1))), "len": length, "k": k,
                "p": rng.choice([8, 16, 31, 64])}
    return {"kind": kind, "n": _log(rng, 100000, 4000000 if kind == "stages" else 8000000), "len": min(length, 200),
            "k": min(k, min(length, 200)), "p": rng.choice([8, 16, 31, 64] if kind != "stages" else [4, 8, 16])}


def _texts(case, seed):
    """Sizes of the suffix sets: log-uniform in [lo, hi], seeded."""
    g = torch.Generator().manual_seed(seed)
    u = torch.rand(case["nsets"], generator=g, dtype=torch.float64).tolist()
    return [int(round(math.exp(math.log(case["lo"]) + x * (math.log(case["hi"]) - math.log(case["lo"]))))) for x in u]


def _suffix_sets(case, seed):
    """All suffixes of case["nsets"] seeded texts, back to back in one arena, and the PE bounds of the sets."""
    # the sizes belong to the case (so that its work does not depend on the seed), the texts to the seed
    sizes = _texts(case, 77)
    chars, offs, lens, pos, n = [], [], [], 0, 0
    begin = [0]
    for s, size in enumerate(sizes):
        ds = d.gen_suffix_strings_device(size, case["max_len"], seed=seed * 1000 + s)
        chars.append(ds.chars[:size])
        offs.append(ds.offsets[:size] + pos)
        lens.append(ds.lengths[:size])
        pos += size
        n += size
        begin.append(n)
    chars.append(torch.zeros(d.PAD, dtype=torch.uint8, device="cuda"))
    ds = d.DeviceStrings(None, chars=torch.cat(chars), offsets=torch.cat(offs), lengths=torch.cat(lens), char_bytes=pos)
    return ds, d.batched_parts(begin, case["p"])


def _outputs(n, p, npe, host=False):
    """The result arrays a program that sorts again and again keeps."""
    import numpy as np
    names = ("local_order", "dp", "perm_index", "perm_pe", "merged_lcp")
    if host:
        out = {k: torch.empty(n, dtype=torch.uint32, pin_memory=True).numpy() for k in names}
    else:
        out = {k: torch.empty(n, dtype=torch.int32, device="cuda") for k in names}
    return dict(out, local_lcp=None, intervals=np.zeros(npe * p, np.uint64), recv_counts=np.zeros(npe, np.uint64))


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx, "p": case.get("p", 0)}
    if kind == "request":
        s["ds"] = d.gen_request_device(ctx, case["n"], seed, case["min_len"], case["max_len"])
    elif kind == "host":
        s["hs"] = d.gen_request(case["n"], seed, case["min_len"], case["max_len"], pinned=True)
    elif kind == "skew":
        s["ds"] = d.gen_dn_device(ctx, case["n"], case["len"], case["k"], seed, case["long_len"], case["long_k"],
                                  case["frac_long"])
    elif kind in ("dn", "ms", "hq", "stages"):
        s["ds"] = d.gen_dn_device(ctx, case["n"], case["len"], case["k"], seed)
    elif kind == "suffix":
        s["ds"], s["parts"] = _suffix_sets(case, seed)
        s["nsets"] = case["nsets"]
    else:
        n, ranges = case["n"], case["ranges"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # LCPs as neighbouring strings have them: geometric, now and then long
        u = torch.rand(n, generator=g, device="cuda").clamp_min(1e-7)
        s["lcps"] = (-20.0 * torch.log(u)).to(torch.int32) * (1 + 9 * (u < 0.01).to(torch.int32))
        s["counts"] = [(r + 1) * n // ranges - r * n // ranges for r in range(ranges)]
        # hashes of one round, a quarter as many, sorted as unsigned words, a block for each of the eight GPUs of a node
        m = n // 4
        s["hcounts"] = [(r + 1) * m // 8 - r * m // 8 for r in range(8)]
        h = torch.randint(-1 << 63, (1 << 63) - 1, (m,), generator=g, device="cuda", dtype=torch.int64)
        s["hashes"] = torch.sort(h).values ^ (-1 << 63)
        s["b"] = [d.golomb_param_hashes(c, 8) for c in s["hcounts"]]
        s["send_bytes"] = torch.zeros(2 * n + 64, dtype=torch.uint8, device="cuda")
        s["send_words"] = torch.zeros(2 * m + 64, dtype=torch.int64, device="cuda")
    if kind in ("request", "dn", "skew"):
        s["out"] = _outputs(case["n"], case["p"], case["p"])
    elif kind == "host":
        s["out"] = _outputs(case["n"], case["p"], case["p"], host=True)
    elif kind == "suffix":
        s["out"] = _outputs(s["ds"].n, case["p"], case["p"] * case["nsets"])
    elif kind == "stages":
        s["send_bytes"] = torch.zeros(case["n"] * (case["len"] + 1), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return s


def _send(buffer, data):
    """What was made for the other side goes into the exchange's send buffer, whose size does not depend on the data."""
    buffer[:data.numel()].copy_(data)
    return buffer


def run(s):
    kind, ctx, p = s["kind"], s["ctx"], s["p"]
    if kind in ("request", "dn", "skew"):
        return dict(d.pd_sort(ctx, s["ds"], p, out=s["out"]))
    if kind == "host":
        return dict(d.pd_sort_host(ctx, s["hs"], p, out=s["out"]))
    if kind == "suffix":
        return dict(d.pd_sort_batched(ctx, s["ds"], s["nsets"], p, s["parts"], out=s["out"]))
    if kind in ("ms", "hq"):
        r = d.ms_sort(ctx, s["ds"], p) if kind == "ms" else d.hq_sort(ctx, s["ds"], p)
        r["chars"] = r["chars"][:r["char_bytes"]]  # what lies behind the strings is padding
        return r
    if kind == "stages":
        ds = s["ds"]
        order, lcp = d.local_sort_lcp(ctx, ds, p)
        dp, rounds = d.dp_prefixes(ctx, ds, order, lcp, p)
        intervals = d.partition(ctx, ds, order, dp, p)
        sent = d.bucket_scatter(ctx, ds, p, order, lcp, dp, intervals)
        merged = d.lcp_merge(ctx, sent["chars"], sent["char_total"], sent["lcp"], sent["counts"], sent["offsets"],
                             sent["char_start"])
        sent["chars"] = _send(s["send_bytes"], sent["chars"][:sent["char_total"]])
        return {"order": order, "lcp": lcp, "dp": dp, "rounds": rounds, "intervals": intervals, "sent": sent,
                "merged": merged}
    coded, per_range = d.varint_encode(ctx, s["lcps"], s["counts"])
    lcps = d.varint_decode(ctx, coded, s["lcps"].numel())
    words, per_block = d.golomb_encode(ctx, s["hashes"], s["hcounts"], s["b"])
    hashes, blocks = d.golomb_decode(ctx, words)
    return {"coded": _send(s["send_bytes"], coded), "per_range": per_range, "lcps": lcps,
            "words": _send(s["send_words"], words), "per_block": per_block, "hashes": hashes, "blocks": blocks}


def _mean_len(case):
    """Mean string length of the request generator: Zipf-like with exponent 1.2 on [min_len, max_len]."""
    ls = range(case["min_len"], case["max_len"] + 1)
    w = [l ** -1.2 for l in ls]
    return sum(l * x for l, x in zip(ls, w)) / sum(w)


def work(case):
    """Bytes of one pass: the string bytes that decide the order (the whole strings where they are copied out), 12 bytes of
    offset and length per string, and every output once.  Nothing is a floating-point operation."""
    kind, n = case["kind"], case.get("n", 0)
    if kind == "wire":
        coded, m = int(1.07 * n), n // 4
        return {"bytes": 2 * (4 * n + coded) + 2 * (8 * m + 6 * m), "flops": 0}
    if kind in ("request", "host"):
        # a string is told apart by its random bytes: about log94(n) of them behind a shared part of a quarter of its length
        need = min(_mean_len(case) + 1, 0.25 * _mean_len(case) + math.log(n) / math.log(94) + 1)
        if kind == "host":
            need = _mean_len(case) + 1  # the whole strings cross the bus
        return {"bytes": n * (need + 12 + 20), "flops": 0}
    if kind == "suffix":
        sizes = _texts(case, 77)
        return {"bytes": sum(sizes) * (1 + 12 + 20), "flops": 0}
    if kind == "skew":
        dist = case["frac_long"] * case["long_k"] + (1 - case["frac_long"]) * case["k"]
        return {"bytes": n * (dist + 12 + 20), "flops": 0}
    if kind == "dn":
        return {"bytes": n * (case["k"] + 12 + 20), "flops": 0}
    if kind == "stages":
        # order and LCP, DP, then the containers: the distinguishing prefixes' own bytes and tags, and the merge's outputs
        return {"bytes": n * (case["k"] + 12 + 8 + 4 + 2 * (7 + 1) + 16 + 20), "flops": 0}
    whole = 2 * (case["len"] + 1) + 12
    return {"bytes": n * (whole + (24 if kind == "ms" else 16)), "flops": 0}


def exact(case, seed):
    """No output is a rounded number: whole numbers and bytes have to be the same as they were."""
    return None
