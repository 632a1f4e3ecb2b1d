"""The GROUP BY work this library is measured on, through its Python entry points.

A case is a dict of plain values:

  kind     "query" (Context.groupby), "batch" (Context.run_batch) or "host"
           (Context.groupby_host, columns and results in pinned host memory)
  rows, ids, zipf    input rows, distinct ids the keys are drawn from, and the
           exponent of the ids' Zipf distribution (0: uniform)
  key      "i32", "u32", "i64", or "pair" (a composite key of two i32 columns)
  cols     value columns, "i32", "i64", "f32" or "f64", separated by commas
  aggs     aggregates, "op:column" or "count"
  nulls    share of absent values in column 0 (0: no validity bitmap)
  sizing   "plain" (the default knobs) or "learned" (the cardinality estimator)
  sort     True: groups in key order, keys spread over their type's range as
           hashed or external ids are.  False: hash-table order (the default);
           the keys are the dense ids of a dimension and the program files
           every group under its id, which is also what makes two runs'
           results comparable.
  misalign rows cut off the front of every column (a slice of a larger table)

A batch draws `queries` shapes from `shapes` (a seed): rows log-uniform in
[2^lo, 2^hi], ids log-uniform in [16, rows / 2], Zipf exponent uniform in
[0, 1.5], 32- or 64-bit keys, SUM and COUNT of one int64 column.

One Context serves every state of a process, as a program keeps one.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from cpu_gpu_coprocess_groupby_agg_b200 import Context, make_knobs
from cpu_gpu_coprocess_groupby_agg_b200 import estimator

_BYTES = {"i32": 4, "u32": 4, "i64": 8, "f32": 4, "f64": 8, "pair": 8}
_TORCH = {"i32": torch.int32, "u32": torch.int32, "i64": torch.int64, "f32": torch.float32, "f64": torch.float64}
_DAYS = 365  # composite keys: (store, day)


def _query(name, rows, ids, zipf=0.0, key="i64", cols="i64", aggs="sum:0,count", nulls=0.0, sizing="plain", sort=False,
           kind="query", misalign=0):
    return {"name": name, "kind": kind, "rows": rows, "ids": ids, "zipf": zipf, "key": key, "cols": cols, "aggs": aggs,
            "nulls": nulls, "sizing": sizing, "sort": sort, "misalign": misalign}


def _batch(name, queries, shapes, lo, hi, sort):
    return {"name": name, "kind": "batch", "queries": queries, "shapes": shapes, "lo": lo, "hi": hi,
            "sizing": "learned", "sort": sort}


def listed():
    return [
        # a dashboard tile over a few thousand recent rows: launches and latency
        _query("tiny", 1 << 12, 64, key="i32", cols="i32"),
        # the small benchmark workload: 2^20 rows over 1024 ids
        _query("small", 1 << 20, 1024, key="i32", cols="i32"),
        # a report by status or region: many rows, few skewed groups, floating
        # averages, an odd row count
        _query("few_groups", (1 << 25) + 35, 64, zipf=1.2, key="i32", cols="f32,f64", aggs="avg:0,sum:1,count"),
        # an ordinary fact table with the default knobs (no estimator loaded),
        # a slice that starts off a 16-byte boundary
        _query("mid_plain", 16_000_003, 200_000, key="i64", aggs="sum:0,count,min:0,max:0", misalign=1),
        # a nullable measure by (store, day), in key order for a report
        _query("nullable_pair", 3_000_017, 50_000, key="pair", cols="i64,f64", aggs="avg:0,count_valid:0,sum:1",
               nulls=0.3, sort=True),
        # deduplicating external ids: nearly every key is its own group
        _query("distinct", 10_000_019, 500_000_000, key="i64", cols="", aggs="count", sort=True),
        # the skewed benchmark workload: 2^26 rows, Zipf 1.0 over 2^20 ids, a
        # wide aggregate list; in key order for a merge downstream
        _query("skewed", 1 << 26, 1 << 20, zipf=1.0, cols="i64,f32", aggs="sum:0,count,min:0,max:0,sum:1",
               sizing="learned", sort=True),
        # the high-cardinality benchmark workload: 2^28 rows over 2^26 ids
        _query("high_card", 1 << 28, 1 << 26, cols="i64,i64", aggs="sum:0,sum:1,count", sizing="learned"),
        # the large serving query, 2^27 rows over 2^24 ids, in key order
        _query("large_sorted", 1 << 27, 1 << 24, sizing="learned", sort=True),
        # the batch benchmark workload: 256 mixed queries in one call
        _batch("batch_256", 256, 4, 12, 24, False),
        # a dashboard's page of small queries in one call, in key order
        _batch("batch_small", 48, 7, 12, 18, True),
        # the rows are in host memory and the groups go back there
        _query("host", 1 << 23, 100_000, key="i32", kind="host", sort=True),
    ]


def draw(rng: random.Random):
    """One more case of the same ranges."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["query"] * 7 + ["batch"] * 2 + ["host"])
    if kind == "batch":
        c = _batch("", log_int(8, 96), rng.randrange(1 << 20), 12, rng.choice([16, 18, 20, 22]), rng.random() < 0.5)
    else:
        rows = log_int(1 << 12, 1 << (23 if kind == "host" else 27))
        ids = log_int(16, max(17, rows // 2))
        key = rng.choice(["i32", "u32", "i64", "i64"] if kind == "host" else ["i32", "u32", "i64", "i64", "pair"])
        cols, aggs = rng.choice([("i64", "sum:0,count"), ("i64", "sum:0,count"), ("i32", "sum:0,count"), ("", "count"),
                                 ("i64,i64", "sum:0,sum:1,count"), ("i64", "sum:0,count,min:0,max:0"),
                                 ("i64,f32", "sum:0,count,min:0,max:0,sum:1")] +
                                ([] if kind == "host" else [("f32,f64", "avg:0,sum:1,count")]))
        nulls = rng.choice([0.0, 0.0, 0.0, 0.2]) if kind == "query" and cols.startswith("i64") else 0.0
        c = _query("", rows, ids, zipf=rng.choice([0.0, round(rng.uniform(0.2, 1.5), 3)]), key=key, cols=cols,
                   aggs=aggs, nulls=nulls, sizing=rng.choice(["plain", "learned"]),
                   sort=kind == "host" or key == "pair" or rng.random() < 0.5, kind=kind,
                   misalign=rng.choice([0, 0, 0, 1]) if kind == "query" and nulls == 0 else 0)
    del c["name"]
    return c


# ---- inputs -----------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _draw_ids(g, rows, ids, zipf):
    """Row ids in [0, ids): uniform, or Zipf over randomly permuted ids."""
    if zipf <= 0:
        return torch.randint(0, ids, (rows,), device="cuda", generator=g)
    cdf = torch.arange(1, ids + 1, device="cuda", dtype=torch.float64).pow_(-zipf).cumsum_(0)
    perm = torch.randperm(ids, device="cuda", generator=g)
    out = torch.empty(rows, dtype=torch.int64, device="cuda")
    for r in range(0, rows, 1 << 25):  # bounded temporaries
        u = torch.rand(min(1 << 25, rows - r), device="cuda", generator=g, dtype=torch.float64) * cdf[-1]
        out[r:r + u.numel()] = perm[torch.searchsorted(cdf, u).clamp_(max=ids - 1)]
    return out


def _key_of_id(ids, key, spread):
    """Key column(s) of dense ids; spread: over the whole range of the type."""
    if key == "pair":
        return ((ids // _DAYS - 1000).to(torch.int32), (ids % _DAYS - 100).to(torch.int32))
    if spread and key == "i64":
        x = ids * 0x2545F4914F6CDD1D + 0x1234567
        ids = (x ^ (x >> 29)) * 0x369DEA0F31A53F85
    elif spread:
        x = (ids * 0x7FEB352D + 0x3C6EF372) & 0xFFFFFFFF
        ids = ((x ^ (x >> 15)) * 0x846CA68B) & 0xFFFFFFFF
    return ids.to(_TORCH[key])


def _column(g, kind, rows):
    if kind in ("f32", "f64"):
        return torch.randn(rows, device="cuda", generator=g, dtype=_TORCH[kind])
    lo, hi = (0, 1000) if kind == "i32" else (-(1 << 31), 1 << 31)
    return torch.randint(lo, hi, (rows,), device="cuda", generator=g, dtype=_TORCH[kind])


def _cols(case):
    return [c for c in case["cols"].split(",") if c]


def _aggs(case):
    return [(a.split(":")[0], int(a.split(":")[1]) if ":" in a else None) for a in case["aggs"].split(",")]


def _is_fp(case, op, col):
    return op == "avg" or (op == "sum" and _cols(case)[col] in ("f32", "f64"))


def _rows(case, seed):
    """(row ids, value columns, presence of column 0 or None) of a query."""
    g = _gen(seed)
    ids = _draw_ids(g, case["rows"], case["ids"], case["zipf"])
    cols = [_column(g, k, case["rows"]) for k in _cols(case)]
    present = torch.rand(case["rows"], device="cuda", generator=g) >= case["nulls"] if case["nulls"] else None
    return ids, cols, present


def _bitmap(present):
    """Arrow validity bitmap: bit i & 7 of byte i >> 3."""
    n = present.numel()
    bits = torch.zeros((n + 7) // 8 * 8, dtype=torch.uint8, device="cuda")
    bits[:n] = present
    weights = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device="cuda")
    return (bits.view(-1, 8) * weights).sum(1, dtype=torch.uint8)


def _shapes(case):
    """The batch's query shapes, 32-bit keys first."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for i in range(case["queries"]):
        n = int(round(2 ** rng.uniform(case["lo"], case["hi"])))
        ids = int(round(math.exp(rng.uniform(math.log(16), math.log(max(17, n // 2))))))
        out.append((i, n, ids, float(rng.uniform(0.0, 1.5)), "i64" if rng.random() < 0.5 else "i32"))
    return sorted(out, key=lambda s: s[4])


def _batch_rows(case, seed, shape):
    i, n, ids, zipf, _ = shape
    g = _gen(seed * 1_000_003 + i)
    return _draw_ids(g, n, ids, zipf), torch.randint(0, 1 << 31, (n,), device="cuda", generator=g)


# ---- what a program keeps ---------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context() -> Context:
    ctx = Context(0)
    estimator.load_default(ctx)
    return ctx


def _offset(t, k):
    """t as a view that starts k elements into its allocation."""
    if not k:
        return t
    room = torch.empty(t.numel() + k, dtype=t.dtype, device=t.device)
    room[k:] = t
    return room[k:]


def _host(t):
    return t.cpu().pin_memory().numpy()


def prepare(case, seed):
    ctx = _context()
    knobs = make_knobs(sizing=case["sizing"], sort_output=int(case["sort"]))
    if case["kind"] == "batch":
        return _prepare_batch(case, seed, ctx, knobs)
    ids, cols, present = _rows(case, seed)
    keys = _key_of_id(ids, case["key"], case["sort"])
    del ids
    aggs, cap = _aggs(case), min(case["rows"], case["ids"]) + 1
    state = {"case": case, "ctx": ctx, "knobs": knobs, "aggs": aggs, "unsigned": case["key"] == "u32"}
    out_types = [torch.float64 if _is_fp(case, op, col) else torch.int64 for op, col in aggs]
    if case["kind"] == "host":
        unsigned = np.uint32 if case["key"] == "u32" else None
        hkeys = _host(keys)
        okeys = torch.zeros(cap, dtype=keys.dtype, pin_memory=True).numpy()
        state["keys"] = hkeys.view(unsigned) if unsigned else hkeys
        state["cols"] = [_host(c) for c in cols]
        state["out"] = (okeys.view(unsigned) if unsigned else okeys,
                        [torch.zeros(cap, dtype=t, pin_memory=True).numpy() for t in out_types])
        return state
    k = case["misalign"]
    state["keys"] = tuple(_offset(x, k) for x in keys) if isinstance(keys, tuple) else _offset(keys, k)
    state["cols"] = [_offset(c, k) for c in cols]
    state["valid"] = [_bitmap(present)] if present is not None else []
    okeys = (tuple(torch.zeros(cap, dtype=torch.int32, device="cuda") for _ in range(2)) if case["key"] == "pair"
             else torch.zeros(cap, dtype=keys.dtype, device="cuda"))
    state["out"] = (okeys, [torch.zeros(cap, dtype=t, device="cuda") for t in out_types])
    state["present"] = [torch.zeros(cap, dtype=torch.uint8, device="cuda") for _ in aggs] if case["nulls"] else []
    if not case["sort"]:
        state["by_id"] = [torch.zeros(case["ids"], dtype=t, device="cuda") for t in out_types]
    return state


def _prepare_batch(case, seed, ctx, knobs):
    shapes = _shapes(case)
    # one arena of result rows for the batch; 32-bit keys come first.  Rows a
    # query leaves unused keep the spare id.
    caps = [min(n, ids) + 1 for _, n, ids, _, _ in shapes]
    n32 = sum(c for c, s in zip(caps, shapes) if s[4] == "i32")
    total, spare = sum(caps), 0 if case["sort"] else sum(s[2] for s in shapes)
    k32 = torch.full((n32,), spare, dtype=torch.int32, device="cuda")
    k64 = torch.full((total - n32,), spare, dtype=torch.int64, device="cuda")
    sums, counts = (torch.zeros(total, dtype=torch.int64, device="cuda") for _ in range(2))
    queries, outs, at, first_id = [], [], 0, 0
    for s, cap in zip(shapes, caps):
        ids, vals = _batch_rows(case, seed, s)
        keys = _key_of_id(ids if case["sort"] else ids + first_id, s[4], case["sort"])
        queries.append((keys, [vals], [("sum", 0), ("count", None)]))
        ok = k32[at:at + cap] if s[4] == "i32" else k64[at - n32:at - n32 + cap]
        outs.append((ok, [sums[at:at + cap], counts[at:at + cap]]))
        at += cap
        first_id += s[2]
    state = {"case": case, "ctx": ctx, "knobs": knobs, "batch": ctx.prepare_batch(queries, outs), "k32": k32,
             "k64": k64, "aggs": [sums, counts], "n32": n32}
    if not case["sort"]:
        state["by_id"] = [torch.zeros(spare + 1, dtype=torch.int64, device="cuda") for _ in range(2)]
    return state


# ---- one pass ---------------------------------------------------------------
def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["kind"] == "batch":
        groups = ctx.run_batch(state["batch"], knobs=state["knobs"])
        if case["sort"]:
            return {"groups": groups, "keys32": state["k32"], "keys64": state["k64"], "aggs": state["aggs"]}
        n32, at32, at64 = state["n32"], state["k32"].long(), state["k64"]
        for table, agg in zip(state["by_id"], state["aggs"]):
            table.index_copy_(0, at32, agg[:n32])
            table.index_copy_(0, at64, agg[n32:])
        return {"groups": groups, "by_id": [t[:-1] for t in state["by_id"]]}
    # result buffers come back whole: rows past the group count stay as prepared
    okeys, oaggs = state["out"]
    if case["kind"] == "host":
        res = ctx.groupby_host(state["keys"], state["cols"], state["aggs"], knobs=state["knobs"], out=state["out"])
        okeys = okeys.view(np.int32) if state["unsigned"] else okeys
        return {"groups": res.n_groups, "keys": [okeys], "aggs": oaggs, "valid": []}
    res = ctx.groupby(state["keys"], state["cols"], state["aggs"], knobs=state["knobs"], out=state["out"],
                      unsigned_keys=state["unsigned"], col_valid=state["valid"], agg_valid=bool(state["valid"]))
    if not case["sort"]:
        at = res.keys.long()
        for table, agg in zip(state["by_id"], res.aggs):
            table.index_copy_(0, at, agg)
        return {"groups": res.n_groups, "by_id": state["by_id"]}
    for table, valid in zip(state["present"], res.valid or []):
        table[:res.n_groups] = valid
    return {"groups": res.n_groups, "keys": list(okeys) if isinstance(okeys, tuple) else [okeys], "aggs": oaggs,
            "valid": state["present"]}


# ---- what a pass cannot do without ------------------------------------------
def _expected_groups(rows, ids, zipf):
    if zipf <= 0:
        return ids * -math.expm1(-rows / ids)
    r = np.unique(np.geomspace(1, ids, 8192).round())
    w = r ** -zipf
    harmonic = np.sum(np.diff(r) * (w[1:] + w[:-1]) / 2) + (w[0] + w[-1]) / 2
    p = -np.expm1(-rows * w / harmonic)
    return float(np.sum(np.diff(r) * (p[1:] + p[:-1]) / 2) + (p[0] + p[-1]) / 2)


def work(case):
    """Every input column read once, every group written once."""
    if case["kind"] == "batch":
        total = 0.0
        for _, n, ids, zipf, key in _shapes(case):
            total += n * (_BYTES[key] + 8) + _expected_groups(n, ids, zipf) * (_BYTES[key] + 16)
        return {"bytes": total, "flops": 0}
    used = {col for op, col in _aggs(case) if op != "count"}
    row = _BYTES[case["key"]] + sum(_BYTES[c] for i, c in enumerate(_cols(case)) if i in used)
    row += 1 / 8 if case["nulls"] else 0
    group = _BYTES[case["key"]] + (9 if case["nulls"] else 8) * len(_aggs(case))
    return {"bytes": case["rows"] * row + _expected_groups(case["rows"], case["ids"], case["zipf"]) * group, "flops": 0}


# ---- the results in 64 bits, by plain torch ---------------------------------
def _order(key_cols, unsigned):
    """The permutation that puts the keys in ascending order."""
    if len(key_cols) == 2:
        k = (key_cols[0].long() << 32) + key_cols[1].long()
    else:
        k = key_cols[0].long()
        k = k & 0xFFFFFFFF if unsigned else k
    return torch.argsort(k)


def _dense(case, ids, cols, present, nids):
    """Per id: row count, every aggregate, every aggregate's validity."""
    n = torch.bincount(ids, minlength=nids)
    aggs, valid = [], []
    for op, col in _aggs(case):
        if op == "count":
            aggs.append(n)
            valid.append((n > 0).to(torch.uint8))
            continue
        x, at, seen = cols[col], ids, n
        if col == 0 and present is not None:
            x, at = x[present], ids[present]
            seen = torch.bincount(at, minlength=nids)
        valid.append((seen > 0).to(torch.uint8))
        fp = x.dtype.is_floating_point
        if op == "count_valid":
            aggs.append(seen)
            continue
        if op in ("min", "max"):
            lim = torch.iinfo(torch.int64)
            t = torch.full((nids,), lim.max if op == "min" else lim.min, dtype=torch.int64, device="cuda")
            t.scatter_reduce_(0, at, x.long(), "amin" if op == "min" else "amax")
        else:
            t = torch.zeros(nids, dtype=torch.float64 if fp else torch.int64, device="cuda")
            t.index_add_(0, at, x.to(t.dtype))
            if op == "avg":
                t = t.double() / seen.double()
        aggs.append(t)
    return n, aggs, valid


def exact(case, seed):
    if case["kind"] == "batch":
        return None  # whole numbers only
    ids, cols, present = _rows(case, seed)
    nids = case["ids"]
    if nids > 4 * case["rows"]:  # few of the ids occur: number those
        names, ids = torch.unique(ids, return_inverse=True)
        nids = names.numel()
    else:
        names = torch.arange(nids, device="cuda")
    n, aggs, valid = _dense(case, ids, cols, present, nids)
    groups = int((n > 0).sum())
    if not case["sort"]:
        return {"groups": groups, "by_id": [torch.where(n > 0, t, torch.zeros_like(t)) for t in aggs]}
    keys = _key_of_id(names[n > 0], case["key"], True)
    keys = list(keys) if isinstance(keys, tuple) else [keys]
    order = _order(keys, case["key"] == "u32")

    def whole(t):  # the result buffer that holds t's groups in key order
        out = torch.zeros(min(case["rows"], case["ids"]) + 1, dtype=t.dtype, device="cuda")
        out[:groups] = t[order]
        return out

    return {"groups": groups, "keys": [whole(k) for k in keys], "aggs": [whole(t[n > 0]) for t in aggs],
            "valid": [whole(v[n > 0]) for v in valid] if case["nulls"] else []}
