"""Performance cases of the group-by path: the calls that its users make, over their range of sizes.

Each case is one call (or one short sequence of calls) through the package's public entry points:
``device.groupby`` (automatic strategy and learned planner), ``device.sort_perm``, ``device.sort_topk``,
``device.unique``, ``device.group_count_distinct``, ``batch.BatchGroupby`` and the host query chain.

  listed()             the cases that are reported by name
  draw(rng)            one more case from the same ranges
  prepare(case, seed)  inputs and kept buffers, on the GPU (host arrays for the chain)
  run(state)           one pass; returns the whole outputs
  work(case)           bytes and operations one pass cannot do without
  exact(case, seed)    what run() returns, by torch in 64 bits
"""

import math

import numpy as np
import torch

from numfast_b200 import batch as nf_batch
from numfast_b200 import device as nf_device
from numfast_b200 import from_numpy
from numfast_b200 import planner as nf_planner

DEVICE = "cuda"
BATCH_MIN_ROWS, BATCH_MAX_ROWS = 1000, 4_000_000
STREAM_KINDS = ("uniform", "zipf", "runs", "clustered")
DTYPES = {"i32": torch.int32, "i64": torch.int64, "f64": torch.float64}
WIDTH = {"i32": 4, "i64": 8, "f64": 8}


def _groupby(name, rows, card, dist="uniform", cols="i32", aggs="sum", nulls=0.0, filtered=False, keep=True):
    """A device.groupby case.  dist: uniform (dense key range), zipf (dense range, skewed), sorted
    (nondecreasing keys) or sparse (keys scattered over the int32 range).  cols: dtypes of the value
    columns.  nulls: fraction of NULL rows in the key and in every column.  filtered: a row filter
    that keeps half the rows.  keep: output buffers kept between calls."""
    return {"name": name, "op": "groupby", "rows": rows, "card": card, "dist": dist, "zipf_s": 1.1, "cols": cols,
            "aggs": aggs, "nulls": nulls, "filtered": filtered, "keep": keep}


def listed():
    return [
        # An interactive query over a small table: launches, read-backs and allocations are the cost.
        _groupby("groupby_10k", 10_007, 250, keep=False),
        # The query chain on host columns: group by a 1,000-value key, order the groups by their sum.
        {"name": "chain_1m", "op": "chain", "rows": 1_000_000, "card": 1000},
        # A report over few groups behind a filter, with NULLs and mixed columns.
        _groupby("groupby_20m_365_filtered", 20_000_003, 365, cols="i32,f64", aggs="sum,min,max", nulls=0.05,
                 filtered=True),
        # The high-cardinality group-by: 100M rows over 10M keys, 5% NULLs per column.
        _groupby("groupby_100m_10m", 100_000_000, 10_000_000, cols="i32,f64", aggs="sum,min,max", nulls=0.05),
        # The same columns under skewed keys (Zipf 1.1 over a 50M domain): a few keys own most rows.
        _groupby("groupby_100m_zipf", 100_000_000, 50_000_000, dist="zipf", cols="i32,f64", aggs="sum,min,max",
                 nulls=0.05),
        # Time-ordered data: keys already nondecreasing, 64-bit integer and float64 measures.
        _groupby("groupby_40m_sorted", 40_000_001, 2_500_000, dist="sorted", cols="i64,f64", aggs="sum"),
        # The learned planner on a stream of inputs of four key distributions (rows, rows/3, rows/9, rows/27).
        {"name": "planner_stream", "op": "stream", "rows": 8_000_009, "card": 400_000},
        # A batch of independent small and middle group-bys in one launch, default tuning.
        {"name": "batch_512", "op": "batch", "queries": 512, "layout": 42},
        # Distinct keys with first row and count over the full int32 range.
        {"name": "unique_200m", "op": "unique", "rows": 200_000_000, "card": 0, "inverse": False},
        # ORDER BY over a float64 column with NULLs, descending.
        {"name": "argsort_30m_f64", "op": "argsort", "rows": 30_000_001, "dtype": "f64", "desc": True, "nulls": 0.05},
        # ORDER BY ... LIMIT 1000 over a large float64 column.
        {"name": "topk_100m_f64", "op": "topk", "rows": 100_000_000, "dtype": "f64", "desc": True, "nulls": 0.05,
         "k": 1000},
        # COUNT(DISTINCT value) per key.
        {"name": "count_distinct_50m", "op": "count_distinct", "rows": 50_000_017, "card": 1_000_000,
         "values": 100_000, "nulls": 0.05},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["groupby"] * 5 + ["chain", "stream", "batch", "unique", "argsort", "argsort", "topk",
                                       "count_distinct"])
    nulls = rng.choice([0.0, 0.05, 0.05, 0.2])
    if op == "groupby":
        dist = rng.choice(["uniform", "uniform", "zipf", "sorted", "sparse"])
        cols = rng.choice(["i32", "f64", "i32,f64", "i64,f64", "i32,i32,f64", "i32,i64,f64,f64"])
        aggs = rng.choice(["sum", "sum,min,max"])
        top = 60_000_000 if cols in ("i32", "f64", "i32,f64") else 20_000_000
        rows = _log_int(rng, 10_000, min(top, 10_000_000) if dist == "sparse" else top)
        c = _groupby("", rows, min(rows, _log_int(rng, 2, 10_000_000)), dist, cols, aggs, nulls,
                     rng.random() < 0.3, rows > 1_000_000)
        c["zipf_s"] = round(rng.uniform(0.5, 2.0), 3)
        c["zipf_s"] = 1.01 if c["zipf_s"] == 1.0 else c["zipf_s"]
    elif op == "chain":
        rows = _log_int(rng, 100_000, 4_000_000)
        c = {"op": op, "rows": rows, "card": _log_int(rng, 10, 20_000)}
    elif op == "stream":
        rows = _log_int(rng, 2_700_000, 12_000_000)
        c = {"op": op, "rows": rows, "card": _log_int(rng, 100, rows)}
    elif op == "batch":
        c = {"op": op, "queries": _log_int(rng, 32, 512), "layout": rng.randrange(1 << 20)}
    elif op == "unique":
        c = {"op": op, "rows": _log_int(rng, 10_000, 100_000_000), "card": rng.choice([0, 0, 1000, 3_000_000]),
             "inverse": rng.random() < 0.4}
    elif op == "argsort":
        c = {"op": op, "rows": _log_int(rng, 10_000, 40_000_000), "dtype": rng.choice(["i32", "i64", "f64"]),
             "desc": rng.random() < 0.5, "nulls": nulls}
    elif op == "topk":
        rows = _log_int(rng, 100_000, 100_000_000)
        c = {"op": op, "rows": rows, "dtype": rng.choice(["i32", "i64", "f64"]), "desc": rng.random() < 0.5,
             "nulls": nulls, "k": _log_int(rng, 1, min(100_000, rows))}
    else:
        rows = _log_int(rng, 100_000, 50_000_000)
        c = {"op": op, "rows": rows, "card": _log_int(rng, 10, rows // 4), "values": _log_int(rng, 2, 1_000_000),
             "nulls": nulls}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs

def _gen(seed, lane=0):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) * 1_000_003 + lane) & 0x7FFFFFFFFFFFFFFF)


# How many distinct keys an input has depends on the case alone: keys and NULL masks come from a
# generator of the case, and the seed turns them (which row holds which draw, which key value stands
# for which rank) and draws every value.  So outputs of two seeds have the same shape.

def _case_gen(case, lane):
    return _gen(case["rows"], 100 + lane)


def _turn_rows(x, seed):
    return None if x is None else torch.roll(x, int(seed) * 2_654_435_761 % max(x.numel(), 1))


def _turn_keys(k, card, seed):
    """Ranks in [0, card) rotated by a step of the seed."""
    return torch.remainder(k + int(seed) * 40_503 % card, card)


def _turn_sparse(k, seed):
    """int32 keys shifted by a step of the seed, wrapping around."""
    return k + (int(seed) * 97_654_321 % (1 << 31))


def _uniform(n, lo, hi, g):
    return torch.randint(lo, hi, (n,), generator=g, dtype=torch.int32, device=DEVICE)


def _zipf(n, s, domain, g):
    """Ranks in [0, domain) by the inverse of the continuous power law x^-s on [1, domain + 1)."""
    u = torch.rand(n, generator=g, dtype=torch.float64, device=DEVICE)
    a = 1.0 - s
    u.mul_((domain + 1.0) ** a - 1.0).add_(1.0).pow_(1.0 / a).floor_().sub_(1.0).clamp_(0, domain - 1)
    return u.to(torch.int32)


def _scatter32(r):
    """A bijective scramble of 32-bit values: dense ranks become keys all over the int32 range."""
    x = r.long()
    for _ in range(2):
        x = ((x ^ (x >> 16)) * 0x45D9F3B) & 0xFFFFFFFF
    x = x ^ (x >> 16)
    return (x - ((x >> 31) << 32)).to(torch.int32)


def _bits(mask):
    """LSB-first bitmap (uint8) of a bool tensor."""
    n = mask.numel()
    m = torch.zeros((n + 7) // 8 * 8, dtype=torch.uint8, device=mask.device)
    m[:n] = mask
    m = m.view(-1, 8)
    out = m[:, 0].clone()
    for i in range(1, 8):
        out |= m[:, i] << i
    return out


def _valid(n, nulls, g):
    if nulls <= 0.0:
        return None
    return torch.rand(n, generator=g, dtype=torch.float32, device=DEVICE) >= nulls


def _keys(case, seed):
    n, card, g = case["rows"], case["card"], _case_gen(case, 1)
    k = _zipf(n, case["zipf_s"], card, g) if case["dist"] == "zipf" else _uniform(n, 0, card, g)
    if case["dist"] == "sorted":
        return torch.sort(k).values + int(seed) % 100_003
    if case["dist"] == "sparse":
        return _turn_rows(_turn_sparse(_scatter32(k), seed), seed)
    return _turn_rows(_turn_keys(k, card, seed) - card // 3, seed)


def _measure(dtype, n, g):
    if dtype == "f64":  # amounts: lognormal(3, 1)
        return torch.randn(n, generator=g, dtype=torch.float64, device=DEVICE).add_(3.0).exp_()
    if dtype == "i64":
        return torch.randint(-(1 << 40), 1 << 40, (n,), generator=g, dtype=torch.int64, device=DEVICE)
    return _uniform(n, -1000, 1001, g)


def _groupby_inputs(case, seed):
    """keys, [(name, dtype, values)], key mask, [column masks], filter mask."""
    n = case["rows"]
    keys = _keys(case, seed)
    cols, masks = [], []
    for i, dt in enumerate(case["cols"].split(",")):
        cols.append(("c%d" % i, dt, _measure(dt, n, _gen(seed, 10 + i))))
        masks.append(_valid(n, case["nulls"], _case_gen(case, 20 + i)))
    masks.append(_valid(n, case["nulls"], _case_gen(case, 2)))
    masks.append(_valid(n, 0.5, _case_gen(case, 3)) if case["filtered"] else None)
    if case["dist"] != "sorted":
        masks = [_turn_rows(m, seed) for m in masks]
    return keys, cols, masks[-2], masks[:-2], masks[-1]


def _order_key(case, seed):
    n, g = case["rows"], _gen(seed, 4)
    if case["dtype"] == "f64":
        k = _measure("f64", n, g)
    elif case["dtype"] == "i64":
        k = _measure("i64", n, g)
    else:
        k = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, dtype=torch.int64, device=DEVICE).to(torch.int32)
    return k, _valid(n, case["nulls"], _gen(seed, 5))


def _stream_inputs(case, seed):
    out = []
    for i, kind in enumerate(STREAM_KINDS):
        n, card, g = max(case["rows"] // 3 ** i, 100_000), max(case["card"] // 3 ** i, 1), _case_gen(case, 30 + i)
        if kind == "uniform":
            k = _turn_rows(_turn_sparse(_scatter32(_uniform(n, 0, card, g)), seed), seed)
        elif kind == "zipf":
            k = _turn_rows(_turn_keys(_zipf(n, 1.2, card, g), card, seed), seed) + 77
        elif kind == "runs":
            starts = torch.rand(n, generator=g, dtype=torch.float32, device=DEVICE) < 0.01
            run = torch.cumsum(starts, 0)
            k = _turn_rows(_turn_keys(_uniform(n, 0, card, g), card, seed)[run], seed)
        else:  # clustered: blocks of 64K rows, each over a window of up to 1,024 scattered keys
            w = min(card, 1024)
            win = _uniform((n + 65535) // 65536, 0, max(card // w, 1), g).repeat_interleave(65536)[:n]
            k = _turn_sparse(_scatter32(win * w + _uniform(n, 0, w, g)), seed)
        out.append((k, _uniform(n, -1000, 1001, _gen(seed, 30 + i))))
    return out


def _batch_layout(case):
    rng = np.random.default_rng(case["layout"])
    nq = case["queries"]
    rows = np.exp(rng.uniform(math.log(BATCH_MIN_ROWS), math.log(BATCH_MAX_ROWS), nq)).astype(np.int64)
    card = np.clip(np.exp(rng.uniform(0.0, np.log(rows))).astype(np.int64), 1, rows)
    zipf = rng.random(nq) < 0.5
    s = rng.uniform(0.5, 2.0, nq)
    s[np.abs(s - 1.0) < 1e-3] = 1.002
    base = rng.integers(-(1 << 30), 1 << 30, nq)
    return rows, card, zipf, s, base


def _batch_inputs(case, seed):
    rows, card, zipf, s, base = _batch_layout(case)
    g = _gen(case["layout"], 40)
    ranks = [_zipf(int(r), float(si), int(c), g) if z else _uniform(int(r), 0, int(c), g)
             for r, c, z, si in zip(rows, card, zipf, s)]
    keys = [_turn_keys(k, int(c), seed) + int(b) for k, c, b in zip(ranks, card, base)]
    off = np.zeros(rows.size + 1, dtype=np.int64)
    off[1:] = np.cumsum(rows)
    return off, torch.cat(keys), _uniform(int(off[-1]), -1000, 1001, _gen(seed, 40))


def _unique_keys(case, seed):
    g = _case_gen(case, 6)
    if case["card"] == 0:
        k = torch.randint(-(1 << 31), 1 << 31, (case["rows"],), generator=g, dtype=torch.int64, device=DEVICE)
        return _turn_rows(_turn_sparse(k.to(torch.int32), seed), seed)
    return _turn_rows(_turn_keys(_uniform(case["rows"], 0, case["card"], g), case["card"], seed), seed)


def _distinct_inputs(case, seed):
    n = case["rows"]
    keys = _turn_keys(_uniform(n, 0, case["card"], _case_gen(case, 7)), case["card"], seed)
    values = _turn_keys(_uniform(n, 0, case["values"], _case_gen(case, 8)), case["values"], seed)
    return (_turn_rows(keys, seed), _turn_rows(values, seed),
            _turn_rows(_valid(n, case["nulls"], _case_gen(case, 9)), seed))


def _chain_inputs(case, seed):
    ranks = np.random.default_rng(case["rows"]).integers(0, case["card"], case["rows"], dtype=np.int32)
    values = np.random.default_rng(int(seed)).integers(-100, 101, case["rows"], dtype=np.int32)
    return {"key": np.roll((ranks + int(seed) % 1009) % case["card"], int(seed)), "v": values}


# ------------------------------------------------------------------ one pass

def prepare(case, seed):
    op = case["op"]
    st = {"op": op, "case": dict(case)}
    if op == "groupby":
        keys, cols, kmask, masks, fmask = _groupby_inputs(case, seed)
        ops = tuple(case["aggs"].split(","))
        st["keys"] = keys
        st["cols"] = [nf_device.DeviceColumn(name, v, ops, None if m is None else _bits(m))
                      for (name, _, v), m in zip(cols, masks)]
        st["kbits"] = None if kmask is None else _bits(kmask)
        st["fbits"] = None if fmask is None else _bits(fmask)
        st["buffers"] = None
        if case["keep"]:
            cap = case["rows"] if case["dist"] == "sparse" else min(case["rows"], case["card"])
            st["buffers"] = nf_device.GroupbyBuffers(cap, st["cols"], torch.device(DEVICE))
    elif op == "chain":
        st["columns"] = _chain_inputs(case, seed)
    elif op == "stream":
        st["inputs"] = _stream_inputs(case, seed)
        st["planner"] = nf_planner.LearnedPlanner.load()
    elif op == "batch":
        off, st["keys"], st["values"] = _batch_inputs(case, seed)
        st["plan"] = nf_batch.BatchGroupby(off)
        st["cap"] = int(off[-1])
    elif op == "unique":
        st["keys"] = _unique_keys(case, seed)
    elif op in ("argsort", "topk"):
        st["keys"], m = _order_key(case, seed)
        st["bits"] = None if m is None else _bits(m)
    else:
        st["keys"], st["values"], m = _distinct_inputs(case, seed)
        st["bits"] = None if m is None else _bits(m)
    return st


def run(st):
    op, case = st["op"], st["case"]
    if op == "groupby":
        r = nf_device.groupby(st["keys"], st["cols"], st["kbits"], buffers=st["buffers"], row_filter=st["fbits"])
        return _groupby_outputs(r, st["cols"])
    if op == "chain":
        t = from_numpy(st["columns"]).query().group("key", {"v": ("sum", "count")}).sort("v.sum", desc=True).compile()
        return {k: np.asarray(v) for k, v in t.to_dict().items()}
    if op == "stream":
        out = []
        for keys, vals in st["inputs"]:
            cols = [nf_device.DeviceColumn("v", vals, ("sum",))]
            r = nf_device.groupby(keys, cols, planner_mode="learned", planner=st["planner"])
            out += _groupby_outputs(r, cols)
        return out
    if op == "batch":
        # The groups of each query are read in query order, whatever place they took in the buffers.
        r = st["plan"].run(st["keys"], st["values"], out_cap=st["cap"])
        ends = torch.cumsum(r.ngroups, 0)
        total = int(ends[-1])
        shift = r.group_offsets - ends + r.ngroups
        at = torch.repeat_interleave(shift, r.ngroups, output_size=total)
        at += torch.arange(total, device=at.device)
        return [r.ngroups, r.ukeys[at], r.sums[at], r.counts[at]]
    if op == "unique":
        r = nf_device.unique(st["keys"], with_inverse=case["inverse"])
        return [r["uniq"], r["first"], r["counts"]] + ([r["inverse"]] if case["inverse"] else [])
    if op == "argsort":
        return nf_device.sort_perm(st["keys"], case["desc"], st["bits"])
    if op == "topk":
        return nf_device.sort_topk(st["keys"], case["k"], case["desc"], st["bits"])
    return list(nf_device.group_count_distinct(st["keys"], st["values"], st["bits"]))


def _groupby_outputs(r, cols):
    out = [r.ukeys, r.counts]
    for c in cols:
        out += [d[c.name] for d in (r.sums, r.mins, r.maxs) if c.name in d]
    return out


# ------------------------------------------------------------------ work

def _expected_groups(rows, card, s=None):
    """Distinct keys expected among `rows` draws (uniform, or the continuous power law of _zipf)."""
    if s is None:
        return card * -math.expm1(-rows / card)
    a = 1.0 - s
    edge = np.unique(np.concatenate([np.arange(1, min(card, 4096) + 1),
                                     np.geomspace(1, card + 1, 20_000).astype(np.int64)])).astype(np.float64)
    lo, hi = edge[:-1], edge[1:]
    p = (hi ** a - lo ** a) / ((card + 1.0) ** a - 1.0) / (hi - lo)  # per key of the interval
    return float(np.sum((hi - lo) * -np.expm1(-rows * p)))


def work(case):
    op = case["op"]
    if op == "groupby":
        dts = case["cols"].split(",")
        maps = (1 + len(dts)) * (case["nulls"] > 0) + case["filtered"]
        live = case["rows"] * (1 - case["nulls"]) ** (1 + len(dts)) * (0.5 if case["filtered"] else 1.0)
        groups = _expected_groups(live, case["card"], case["zipf_s"] if case["dist"] == "zipf" else None)
        aggs = case["aggs"].split(",")
        per = 16 + sum(8 * ("sum" in aggs) + WIDTH[d] * (("min" in aggs) + ("max" in aggs)) for d in dts)
        b = case["rows"] * (4 + sum(WIDTH[d] for d in dts) + maps / 8) + groups * per
        return {"bytes": b, "flops": live * len(dts) * len(aggs)}
    if op == "chain":
        return {"bytes": 8 * case["rows"] + 24 * _expected_groups(case["rows"], case["card"]),
                "flops": case["rows"]}
    if op == "stream":
        rows = [max(case["rows"] // 3 ** i, 100_000) for i in range(len(STREAM_KINDS))]
        cards = [max(case["card"] // 3 ** i, 1) for i in range(len(STREAM_KINDS))]
        g = [_expected_groups(n, c, 1.2 if k == "zipf" else None) for n, c, k in zip(rows, cards, STREAM_KINDS)]
        return {"bytes": 8 * sum(rows) + 24 * sum(g), "flops": sum(rows)}
    if op == "batch":
        rows, card, zipf, s, _ = _batch_layout(case)
        g = sum(_expected_groups(int(r), int(c), float(si) if z else None)
                for r, c, z, si in zip(rows, card, zipf, s))
        return {"bytes": 8 * int(rows.sum()) + 24 * g, "flops": int(rows.sum())}
    if op == "unique":
        g = _expected_groups(case["rows"], case["card"] or 1 << 32)
        return {"bytes": 4 * case["rows"] * (2 if case["inverse"] else 1) + 16 * g, "flops": case["rows"]}
    if op == "argsort":
        return {"bytes": case["rows"] * (WIDTH[case["dtype"]] + 4 + (case["nulls"] > 0) / 8), "flops": case["rows"]}
    if op == "topk":
        return {"bytes": case["rows"] * (WIDTH[case["dtype"]] + (case["nulls"] > 0) / 8) + 4 * case["k"],
                "flops": case["rows"]}
    return {"bytes": case["rows"] * (8 + (case["nulls"] > 0) / 8) +
            16 * _expected_groups(case["rows"], case["card"]), "flops": case["rows"]}


# ------------------------------------------------------------------ exact results

def _sum_by(code, v, ng):
    """Sums per group code: int64 for integers; for float64 the sum of two exact integer parts
    (20 binary places, then 32 more), so the order of the rows does not matter."""
    if v.dtype != torch.float64:
        return torch.zeros(ng, dtype=torch.int64, device=v.device).index_add_(0, code, v.long())
    x = v * float(1 << 20)
    hi = x.floor()
    lo = ((x - hi) * float(1 << 32)).long()
    hs = torch.zeros(ng, dtype=torch.int64, device=v.device).index_add_(0, code, hi.long())
    ls = torch.zeros_like(hs).index_add_(0, code, lo)
    hs += ls >> 32
    return hs.double() / float(1 << 20) + (ls & 0xFFFFFFFF).double() / float(1 << 52)


def _group_exact(keys, cols, live):
    """[ukeys, counts, then per column its aggregates] of the live rows."""
    if live is not None:
        keys = keys[live]
    uk, code, counts = torch.unique(keys, return_inverse=True, return_counts=True)
    out = [uk.long(), counts]
    for v, aggs in cols:
        if live is not None:
            v = v[live]
        if "sum" in aggs:
            out.append(_sum_by(code, v, uk.numel()))
        for name, red in (("min", "amin"), ("max", "amax")):
            if name in aggs:
                z = torch.zeros(uk.numel(), dtype=v.dtype, device=v.device)
                out.append(z.scatter_reduce_(0, code, v, red, include_self=False))
    return out


def _both(*masks):
    m = None
    for x in masks:
        if x is not None:
            m = x if m is None else m & x
    return m


def _order_exact(keys, desc, valid):
    """Stable order; descending keeps input order among ties; NULL rows last in input order."""
    if valid is None:
        return torch.sort(keys, stable=True, descending=desc).indices.to(torch.int32)
    pos = torch.nonzero(valid).flatten()
    order = torch.sort(keys[pos], stable=True, descending=desc).indices
    return torch.cat([pos[order], torch.nonzero(~valid).flatten()]).to(torch.int32)


def exact(case, seed):
    op = case["op"]
    if op == "groupby":
        keys, cols, kmask, masks, fmask = _groupby_inputs(case, seed)
        return _group_exact(keys, [(v, case["aggs"].split(",")) for _, _, v in cols], _both(kmask, fmask, *masks))
    if op == "chain":
        c = _chain_inputs(case, seed)
        uk, code = np.unique(c["key"], return_inverse=True)
        sums = np.zeros(uk.size, dtype=np.int64)
        np.add.at(sums, code, c["v"])
        order = np.argsort(-sums, kind="stable")
        return {"key": uk[order].astype(np.int64), "v.sum": sums[order], "v.count": np.bincount(code)[order]}
    if op == "stream":
        out = []
        for k, v in _stream_inputs(case, seed):
            out += _group_exact(k, [(v, ("sum",))], None)
        return out
    if op == "batch":
        off, keys, values = _batch_inputs(case, seed)
        rows = torch.from_numpy(np.diff(off)).to(DEVICE)
        query = torch.repeat_interleave(torch.arange(rows.numel(), device=DEVICE), rows)
        u, code, counts = torch.unique((query << 32) + (keys.long() + (1 << 31)), return_inverse=True,
                                       return_counts=True)
        ng = torch.bincount(u >> 32, minlength=rows.numel())
        return [ng, (u & 0xFFFFFFFF) - (1 << 31), _sum_by(code, values, u.numel()), counts]
    if op == "unique":
        keys = _unique_keys(case, seed)
        uk, code, counts = torch.unique(keys, return_inverse=True, return_counts=True)
        first = torch.full((uk.numel(),), keys.numel(), dtype=torch.int64, device=DEVICE)
        first.scatter_reduce_(0, code, torch.arange(keys.numel(), device=DEVICE), "amin")
        return [uk, first.to(torch.int32), counts] + ([code.to(torch.int32)] if case["inverse"] else [])
    if op == "argsort":
        return _order_exact(*_order_args(case, seed))
    if op == "topk":
        return _order_exact(*_order_args(case, seed))[:case["k"]].clone()
    keys, values, valid = _distinct_inputs(case, seed)
    if valid is not None:
        keys, values = keys[valid], values[valid]
    pairs = torch.unique((keys.long() << 32) + values.long())
    uk, counts = torch.unique_consecutive(pairs >> 32, return_counts=True)
    return [uk, counts]


def _order_args(case, seed):
    keys, valid = _order_key(case, seed)
    return keys, case["desc"], valid
