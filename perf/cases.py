"""The joins that this framework is timed on, each through the entry points that a program calls.

Every case joins a relation of unique keys with one whose rows match it at most once, so a program that
wants "the other side's value beside each of my rows" (a lookup join) gets a well-defined column. The
engine writes its pairs in an unspecified order; `run` places each pair's value at its row, as such a
program does, and returns the aligned column(s) with the exact match count. Rows without a partner hold
-1. Values are row numbers, as in the benchmark's inputs. Outputs are whole numbers and have to be equal.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "brig-join_b200"))
import brig_join as bj  # noqa: E402

M = 1_000_000


def _join(name=None, *, n_r, n_s, match, zipf=0.0, bloom=0.0, mode=0, key=False, fact="s"):
    """One device join of n_r unique keys (the generator's R) with n_s rows (its S), `match` of which find
    a partner, drawn uniformly or Zipf-skewed. bloom: filter bits per key (0: no filter); mode: 0 radix
    bits, 1 key % 512 and the reference's second level; key: the pairs' keys come back too; fact: "s"
    joins unique R with S, "r" gives the skewed relation as R and the unique one as S."""
    c = {"kind": "join", "n_r": n_r, "n_s": n_s, "match": match, "zipf": zipf, "bloom": bloom, "mode": mode,
         "key": key, "fact": fact}
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest joins of the batch and serving workloads, one at a time: latency and launches.
        _join("tiny 4K x 16K", n_r=4096, n_s=16384, match=0.1),
        # A served request of the smallest size, odd sizes, filter on.
        _join("small 65K x 262K filter", n_r=65_537, n_s=262_147, match=0.1, bloom=10.0),
        # An ordinary dimension lookup with skewed matches, keys returned with the pairs.
        _join("1M x 4M zipf keys", n_r=1_000_003, n_s=4_000_037, match=0.3, zipf=1.0, key=True),
        # The plain single join of the benchmark's first configuration.
        _join("16M x 16M filter", n_r=1 << 24, n_s=1 << 24, match=0.1, bloom=10.0),
        # The reference's partition layout (key % 512, second level sized as the reference does).
        _join("10M x 20M modulo filter", n_r=10_000_019, n_s=20_000_003, match=0.1, bloom=10.0, mode=1),
        # A foreign-key join: every row matches, no filter.
        _join("4M x 16M all match", n_r=4_000_037, n_s=16_000_057, match=1.0),
        # The skewed relation given as R: hot keys, partitions far above the table capacity.
        _join("16M zipf R x 2M", n_r=2_000_003, n_s=16_000_057, match=0.5, zipf=1.0, fact="r"),
        # The selectivity sweep's shape: few matches, filter of the sweep's middle size.
        _join("64M x 1G 1% filter", n_r=1 << 26, n_s=1 << 30, match=0.01, bloom=10.0),
        # The headline join of the benchmark.
        _join("640M x 640M filter", n_r=640 * M, n_s=640 * M, match=0.1, bloom=10.0),
        # Uneven joins in one pipeline: |R| log-uniform in [4K, 16M], |S| = 4|R|, Zipf matches, replayed graph.
        {"name": "batch of 64", "kind": "batch", "joins": 64, "sizes": 3, "lo": 4096, "hi": 1 << 24, "match": 0.1,
         "zipf": 1.0, "bloom": 10.0},
        # The whole call over host arrays (pinned), copies included.
        {"name": "host 12M x 4M filter", "kind": "host", "n_r": 12_000_017, "n_s": 4_000_037, "match": 0.1,
         "bloom": 10.0},
        # Requests of the serving loop's small sizes on device-resident relations, answers back on the host.
        {"name": "serve 12 requests", "kind": "serve", "requests": 12, "sizes": 5, "lo": 1 << 16, "hi": 1 << 20,
         "bloom": 10.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["join", "batch", "host", "serve"], [0.7, 0.1, 0.1, 0.1])[0]
    if kind == "batch":
        return {"kind": "batch", "joins": rng.randint(6, 64), "sizes": rng.randrange(1 << 20), "lo": 4096,
                "hi": _log(rng, 1 << 20, 1 << 24), "match": rng.choice([0.05, 0.1, 0.3]), "zipf": rng.choice([0.0, 1.0]),
                "bloom": rng.choice([0.0, 8.0, 10.0])}
    if kind == "host":
        return {"kind": "host", "n_r": _log(rng, 1 << 16, 12 * M), "n_s": _log(rng, 1 << 16, 4 * M),
                "match": rng.choice([0.01, 0.1, 0.3]), "bloom": rng.choice([0.0, 10.0])}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(4, 16), "sizes": rng.randrange(1 << 20), "lo": 1 << 16,
                "hi": _log(rng, 1 << 18, 1 << 20), "bloom": rng.choice([0.0, 10.0])}
    fact = rng.choice(["s", "s", "s", "r"])
    zipf = rng.choice([0.0, 0.0, 1.0])
    mode = rng.choice([0, 0, 0, 1])
    bloom = rng.choice([0.0, 8.0, 10.0, 10.0, 14.0])
    # the costlier options (skew, modulo layout, no filter) stay below the largest listed join's time
    top = 32 * M if zipf else 100 * M if mode else 250 * M if not bloom else 600 * M
    n_r = _log(rng, 4096, top)
    n_s = max(4096, min(int(n_r * rng.uniform(0.25, 16.0)), top, 800 * M - n_r)) | 1
    match = rng.choice([0.001, 0.01, 0.1, 0.3, 0.6, 1.0])
    if match * n_s > 20 * M:
        match = round(20 * M / n_s, 4)
    return _join(n_r=n_r, n_s=n_s, match=match, zipf=zipf, bloom=bloom, mode=mode, key=rng.random() < 0.25, fact=fact)


def _sizes(case):
    """[(unique rows, other rows, match share)] of a batch or a set of requests."""
    r = random.Random(case["sizes"])
    out = []
    for _ in range(case.get("joins") or case["requests"]):
        n = _log(r, case["lo"], case["hi"])
        if case["kind"] == "batch":
            out.append((n, 4 * n, case["match"]))
        else:
            out.append((n, n * r.choice([1, 4]), r.choice([0.01, 0.1])))
    return out


def _slots(match, n):
    """Output slots of a join that expects `match` of n rows to find a partner."""
    return int(match * n) + 64


def _config(case):
    cfg = dict(partition_mode=case.get("mode", 0))
    if cfg["partition_mode"]:
        cfg["partition_size"] = 512
    if case["bloom"]:
        cfg.update(use_bloom=1, bloom_bits_per_key=case["bloom"])
    return cfg


def _gen(seed, n_r, n_s, match, zipf=0.0):
    t = [torch.empty(n, dtype=torch.int32, device="cuda") for n in (n_r, n_r, n_s, n_s)]
    bj.gen_device(seed, n_r, n_s, match, zipf, *t)
    return t


def _prepare_join(case, seed):
    n_r, n_s = case["n_r"], case["n_s"]
    uk, uv, fk, fv = _gen(seed, n_r, n_s, case["match"], case["zipf"])
    slots = _slots(case["match"], n_s)
    left, right = ((uk, uv), (fk, fv)) if case["fact"] == "s" else ((fk, fv), (uk, uv))
    return {"kind": "join", "handle": bj.Join(**_config(case)), "left": left, "right": right, "rows": n_s,
            "fact": case["fact"], "slots": slots,
            "out_r": torch.empty(slots, dtype=torch.int32, device="cuda"),
            "out_s": torch.empty(slots, dtype=torch.int32, device="cuda"),
            "out_k": torch.empty(slots, dtype=torch.int32, device="cuda") if case["key"] else None,
            "count": torch.zeros(1, dtype=torch.int64, device="cuda"),
            "col": torch.empty(n_s + 1, dtype=torch.int32, device="cuda"),
            "keys": torch.empty(n_s + 1, dtype=torch.int32, device="cuda") if case["key"] else None}


def _prepare_batch(case, seed):
    sizes = _sizes(case)
    rows = sum(n_s for _, n_s, _ in sizes)
    slots = sum(_slots(m, n_s) for _, n_s, m in sizes)
    out_r = torch.empty(slots, dtype=torch.int32, device="cuda")
    out_s = torch.empty(slots, dtype=torch.int32, device="cuda")
    counts = torch.zeros(len(sizes), dtype=torch.int64, device="cuda")
    items, base, at = [], 0, 0
    for i, (n_r, n_s, m) in enumerate(sizes):
        rk, rv, sk, sv = _gen(seed * 1000 + i, n_r, n_s, m, case["zipf"])
        sv += base  # row of the joins' S rows laid end to end
        cap = _slots(m, n_s)
        items.append(dict(r_key=rk, r_val=rv, n_r=n_r, s_key=sk, s_val=sv, n_s=n_s, out_r=out_r[at:at + cap],
                          out_s=out_s[at:at + cap], capacity=cap, d_count=counts[i:i + 1]))
        base += n_s
        at += cap
    return {"kind": "batch", "handle": bj.Join(use_cuda_graph=1, **_config(case)), "items": items, "rows": rows,
            "out_r": out_r, "out_s": out_s, "count": counts,
            "col": torch.empty(rows + 1, dtype=torch.int32, device="cuda")}


def _pinned(n, dtype=torch.int32):
    return torch.empty(n, dtype=dtype, pin_memory=True)


def _u32(t):
    return t.numpy().view(np.uint32)


def _prepare_host(case, seed):
    n_r, n_s = case["n_r"], case["n_s"]
    host = []
    for t in _gen(seed, n_r, n_s, case["match"]):
        h = _pinned(t.numel())
        h.copy_(t)
        host.append(h)
    slots = _slots(case["match"], n_s)
    out = (_pinned(slots), _pinned(slots))
    return {"kind": "host", "handle": bj.Join(**_config(case)), "in": host, "out": out, "slots": slots,
            "col": torch.empty(n_s, dtype=torch.int32)}


def _prepare_serve(case, seed):
    sizes = _sizes(case)
    reqs, base = [], 0
    for i, (n_r, n_s, m) in enumerate(sizes):
        rk, rv, sk, sv = _gen(seed * 1000 + i, n_r, n_s, m)
        sv += base
        cap = _slots(m, n_s)
        reqs.append((rk, rv, sk, sv, cap, (_pinned(cap), _pinned(cap))))
        base += n_s
    return {"kind": "serve", "server": bj.Server(**_config(case)), "reqs": reqs,
            "col": torch.empty(base, dtype=torch.int32)}


def prepare(case, seed):
    return {"join": _prepare_join, "batch": _prepare_batch, "host": _prepare_host,
            "serve": _prepare_serve}[case["kind"]](case, seed)


def _place(col, rows, values):
    """col[row] = value of every pair; the slots past the last pair hold the spare row at the end."""
    col.fill_(-1)
    return col.scatter_(0, rows.long(), values)


def _run_join(s):
    rows, values = (s["out_s"], s["out_r"]) if s["fact"] == "s" else (s["out_r"], s["out_s"])
    rows.fill_(s["rows"])
    (rk, rv), (sk, sv) = s["left"], s["right"]
    s["handle"].run(rk, rv, rk.numel(), sk, sv, sk.numel(), s["out_r"], s["out_s"], s["slots"], out_key=s["out_k"],
                    d_count=s["count"])
    out = {"column": _place(s["col"], rows, values)[:s["rows"]], "count": s["count"]}
    if s["keys"] is not None:
        out["keys"] = _place(s["keys"], rows, s["out_k"])[:s["rows"]]
    return out


def _run_batch(s):
    s["out_s"].fill_(s["rows"])
    s["handle"].run_batch(s["items"])
    return {"column": _place(s["col"], s["out_s"], s["out_r"])[:s["rows"]], "count": s["count"]}


def _run_host(s):
    count, r, v = s["handle"].run_host(*[_u32(t) for t in s["in"]], capacity=s["slots"],
                                       out=(_u32(s["out"][0]), _u32(s["out"][1]), None))
    n = min(count, s["slots"])
    s["col"].fill_(-1)
    s["col"][s["out"][1][:n]] = s["out"][0][:n]
    return {"column": s["col"], "count": count}


def _run_serve(s):
    tickets = [s["server"].submit(rk, rv, sk, sv, capacity=cap, out=(_u32(out[0]), _u32(out[1])), on_device=True)
               for rk, rv, sk, sv, cap, out in s["reqs"]]
    s["col"].fill_(-1)
    counts = []
    for t, (_, _, _, _, cap, out) in zip(tickets, s["reqs"]):
        res, _, _ = s["server"].poll(t)
        n = min(res.count, cap)
        counts.append(res.count)
        s["col"][out[1][:n]] = out[0][:n]
    return {"column": s["col"], "count": np.array(counts, np.int64)}


def run(s):
    return {"join": _run_join, "batch": _run_batch, "host": _run_host, "serve": _run_serve}[s["kind"]](s)


def work(case):
    """Keys and values of both relations read once, pairs (and keys) and the aligned columns written once."""
    sizes = [(case["n_r"], case["n_s"], case["match"])] if "n_r" in case else _sizes(case)
    words = 3 if case.get("key") else 2
    return {"bytes": float(sum(8 * (r + s) + 4 * words * int(m * s) + 4 * (words - 1) * s for r, s, m in sizes)),
            "flops": 0.0}


def tolerance(case):
    return "exact"
