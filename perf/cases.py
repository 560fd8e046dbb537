"""The work that users of the framework have it do, as cases that can be timed:
range filters, group-bys, the reference's sort / group / aggregate chain, joins
and a batch of mixed queries, each through the public entry points, from a few
thousand rows to the sizes of the benchmark configurations.

listed() gives the standing cases, draw() more of the same ranges.  Where the
operators leave an order open (rows of equal key in a join's output), the
inputs are such that every order gives the same output.
"""
from __future__ import annotations

import math

import torch

from query_on_opencl_fpga_gb300 import batch as qbatch
from query_on_opencl_fpga_gb300 import datagen
from query_on_opencl_fpga_gb300.api import Context

I32_MIN = -(2 ** 31)
SUM = 0
CATEGORIES = 1000  # values of a payload column, as in every benchmark configuration

_ctx = None


def context() -> Context:
    """The process's context: a program makes one per thread and keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = Context()
    return _ctx


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def listed():
    return [
        # A selection on a small table: what one call costs when the data costs nothing.
        {"name": "filter_4k", "op": "filter", "n": 4097, "sel": 0.1},
        # The plain filter of the benchmark: 16M rows, a tenth selected.
        {"name": "filter_16m", "op": "filter", "n": 1 << 24, "sel": 0.1},
        # The reference's own layout: a ragged table of records, a larger share kept.
        {"name": "filter_rec_5m", "op": "filter_rec", "n": 5_000_011, "sel": 0.4},
        # SUM and COUNT by a short list of categories over a small table.
        {"name": "groupby_10k", "op": "groupby", "n": 10_007, "groups": 512, "fused": False},
        # The benchmark's group-by: 64M rows, Zipf over a million groups.
        {"name": "groupby_64m", "op": "groupby", "n": 1 << 26, "groups": 1 << 20, "fused": False},
        # Filter and aggregation in one call, on a ragged table of middling size.
        {"name": "fused_24m", "op": "groupby", "n": 24_000_001, "groups": 1 << 20, "fused": True},
        # Group-by on identifiers spread over all 32 bits (hashed ids).
        {"name": "groupby_ids_8m", "op": "groupby_ids", "n": 8_000_003, "groups": 1_000_000},
        # The reference's chain on records: sort by key, group starts, SUM per group.
        {"name": "records_16m", "op": "records", "n": 16_777_213, "groups": 1 << 20, "span": 1 << 20},
        # A lookup of a small fact table in a small dimension table.
        {"name": "join_20k", "op": "join", "nr": 1_250, "ns": 20_011},
        # The benchmark's join: 16M build rows, 256M probe rows, 30 % kept, sorted output.
        {"name": "join_256m", "op": "join", "nr": 1 << 24, "ns": 1 << 28},
        # Keys in a few dense regions and some very frequent ones.
        {"name": "join_skew_32m", "op": "join_skew", "nr": 4_000_000, "ns": 32_000_000},
        # A report of many queries of uneven sizes, replayed as one graph.
        {"name": "batch_24", "op": "batch", "each": 6, "lo": 4096, "hi": 1 << 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["filter", "filter_rec", "groupby", "groupby_ids", "records", "join", "join_skew", "batch"])
    if op in ("filter", "filter_rec"):
        return {"op": op, "n": _log(rng, 4096, 1 << 24), "sel": round(rng.uniform(0.02, 0.9), 3)}
    if op == "groupby":
        n = _log(rng, 4096, 1 << 26)
        return {"op": op, "n": n, "groups": _log(rng, 64, min(n // 4, 1 << 20)), "fused": rng.random() < 0.5}
    if op == "groupby_ids":
        n = _log(rng, 4096, 1 << 25)
        return {"op": op, "n": n, "groups": _log(rng, 64, min(n // 4, 1 << 20))}
    if op == "records":
        n = _log(rng, 4096, 1 << 26)
        groups = _log(rng, 64, n // 4)
        return {"op": op, "n": n, "groups": groups, "span": _log(rng, groups, 2 ** 31 - 1)}
    if op == "join":
        ns = _log(rng, 4096, 1 << 28)
        return {"op": op, "nr": max(16, ns // _log(rng, 8, 64)), "ns": ns}
    if op == "join_skew":
        ns = _log(rng, 65536, 1 << 26)
        return {"op": op, "nr": max(1024, ns // _log(rng, 8, 32)), "ns": ns}
    lo = _log(rng, 4096, 65536)
    return {"op": op, "each": rng.randint(1, 6), "lo": lo, "hi": _log(rng, 1 << 20, 1 << 24)}


# --------------------------------------------------------------------------
# Inputs.  The number of rows or groups that come out is the same for every
# seed (which rows, keys and values they are is not), so that results of
# different inputs have one shape.
# --------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _perm(n, seed):
    return torch.randperm(n, generator=_gen(seed), device="cuda")


def _below(n, m, seed):
    """int64 uniform in [0, m)."""
    return torch.randint(0, m, (n,), generator=_gen(seed), dtype=torch.int64, device="cuda")


def _category(key):
    """A payload column that the key determines (the product's category beside its id)."""
    k = key.to(torch.int64) & 0xFFFFFFFF
    return (((k * 2654435761) & 0xFFFFFFFF) >> 7) % CATEGORIES


def _filter_in(n, sel, seed):
    """Keys uniform over [0, 2^31) of which the share `sel` is at most `hi`."""
    hi = int(sel * 2 ** 31)
    keep = _perm(n, seed + 2) < int(n * sel)
    key = torch.where(keep, _below(n, hi + 1, seed), hi + 1 + _below(n, 2 ** 31 - 1 - hi, seed + 1))
    return {"key": key.to(torch.int32), "pay": datagen.uniform_i32(n, 0, CATEGORIES, seed + 3, "cuda"),
            "lo": I32_MIN, "hi": hi}


def _groupby_in(n, groups, seed):
    """Zipf(1.0) keys, every group present (also among the rows that the fused form keeps)."""
    d = datagen.config1_groupby(n, groups, seed=seed, device="cuda")
    at = _perm(n, seed + 5)[:groups]
    d["key"][at] = torch.arange(groups, dtype=torch.int32, device="cuda")
    d["val2"][at] = d["val2"][at] // 2
    return d


def _ids(groups, span, seed):
    """`groups` distinct keys spread over [0, span), in no order."""
    step = span // groups
    i = torch.arange(groups, device="cuda") * step + _below(groups, step, seed)
    return i[_perm(groups, seed + 1)]


def _id_keys(n, groups, span, seed):
    """n keys uniform over such a set, every one of them present."""
    pick = torch.cat([torch.arange(groups, device="cuda"), _below(n - groups, groups, seed + 2)])
    return _ids(groups, span, seed)[pick[_perm(n, seed + 3)]]


def _join_in(nr, ns, seed):
    """R: a permutation of [0, nr).  S: four fifths of the rows have a key of R, 30 % of the keys (and
    of those rows) a category that the filter keeps, the other rows keys above R's."""
    rank = _perm(nr, seed + 4)                      # the key's place among the categories
    kept = (3 * nr) // 10
    by_rank = torch.argsort(rank)
    role = _perm(ns, seed + 5)
    n_in, n_hit = (4 * ns) // 5, (24 * ns) // 100
    r = torch.where(role < n_hit, _below(ns, kept, seed + 6), kept + _below(ns, nr - kept, seed + 7))
    out = max(nr, 1 << 24) + _below(ns, 2 ** 31 - max(nr, 1 << 24), seed + 8)
    inside = role < n_in
    skey = torch.where(inside, by_rank[r], out)
    spay = torch.where(inside, torch.where(r < kept, r * 300 // kept, 300 + (r - kept) * 700 // (nr - kept)),
                       _category(out))
    return {"rkey": _perm(nr, seed).to(torch.int32), "rpay": datagen.uniform_i32(nr, 0, CATEGORIES, seed + 1, "cuda"),
            "skey": skey.to(torch.int32), "spay": spay.to(torch.int32), "slo": I32_MIN, "shi": 299}


def _skew_hits(nr, ns):
    """Output rows of the skewed join: about what the mixture gives by itself."""
    return int(ns * (0.006 - 0.2 * math.expm1(-6e-8 * nr)))


def _skew_in(nr, ns, seed):
    """The skewed keys of the benchmark (8 Gaussians and 5 % heavy hitters), a few probe rows
    exchanged for others until _skew_hits of them come out."""
    d = datagen.config4_skewed(nr, ns, seed=seed, device="cuda")
    rk = torch.sort(d["rkey"])[0]

    def hits(k):
        at = torch.searchsorted(rk, k).clamp_(max=nr - 1)
        return (rk[at] == k) & (_category(k) < 300)

    hit = hits(d["skey"])
    yes, no = torch.nonzero(hit).reshape(-1), torch.nonzero(~hit).reshape(-1)
    more = _skew_hits(nr, ns) - yes.numel()
    if yes.numel() == 0:
        raise ValueError("no probe row matches")
    src, dst = (yes, no) if more > 0 else (no, yes)
    dst = dst[_perm(dst.numel(), seed + 21)[: abs(more)]]
    d["skey"][dst] = d["skey"][src[_below(dst.numel(), src.numel(), seed + 22)]]
    d["spay"] = _category(d["skey"]).to(torch.int32)
    return d


def _batch_queries(case, seed):
    """`each` queries of every operator, row counts log-uniform in [lo, hi]."""
    each, lo, hi = case["each"], case["lo"], case["hi"]
    rng = torch.Generator().manual_seed(4 * each + 1)  # sizes belong to the case, data to the seed
    counts = torch.zeros(4 * each, dtype=torch.int64, device="cuda")
    qs = []
    for i in range(4 * each):
        op, s = i % 4, 1000 * seed + 10 * i
        n = int(round(lo * (hi / lo) ** float(torch.rand(1, generator=rng))))
        q = {"op": op, "n": n, "variant": -1, "count": counts[i: i + 1]}
        if op == qbatch.OP_FILTER:
            d = _filter_in(n, 0.1, s)
            q.update(inp=[d["key"], d["pay"]], lo=d["lo"], hi=d["hi"], n2=0, cap=n)
            q["out"] = [torch.zeros((n, 2), dtype=torch.int32, device="cuda")]
        elif op == qbatch.OP_JOIN:
            nr = max(n // 16, 16)
            d = _join_in(nr, n, s)
            q.update(inp=[d["rkey"], d["rpay"], d["skey"], d["spay"]], lo=d["slo"], hi=d["shi"], n2=nr, cap=n)
            q["out"] = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3)]
        else:
            d = datagen.config1_groupby(n, 1 << 20, seed=s, device="cuda")
            cap = min(n, 1 << 20)
            q.update(inp=[d["key"], d["val"], d["val2"]], lo=d["lo2"], hi=d["hi2"], n2=1 << 20, cap=cap)
            q["out"] = [torch.zeros(cap, dtype=t, device="cuda") for t in (torch.int32, torch.int64, torch.int64)]
        qs.append(q)
    return qs, counts


def _inputs(case, seed):
    op = case["op"]
    if op == "filter":
        return _filter_in(case["n"], case["sel"], seed)
    if op == "filter_rec":
        d = _filter_in(case["n"], case["sel"], seed)
        return {"rec": datagen.records(d["key"]), "lo": d["lo"], "hi": d["hi"]}
    if op == "groupby":
        return _groupby_in(case["n"], case["groups"], seed)
    if op == "groupby_ids":
        key = _id_keys(case["n"], case["groups"], 2 ** 32, seed)
        key = torch.where(key >= 2 ** 31, key - 2 ** 32, key).to(torch.int32)
        return {"key": key, "val": datagen.uniform_i32(case["n"], 0, CATEGORIES, seed + 4, "cuda")}
    if op == "records":
        key = _id_keys(case["n"], case["groups"], case["span"], seed).to(torch.int32)
        return {"rec": datagen.records(key, datagen.uniform_i32(case["n"], 0, CATEGORIES, seed + 4, "cuda"))}
    if op == "join":
        return _join_in(case["nr"], case["ns"], seed)
    return _skew_in(case["nr"], case["ns"], seed)


def prepare(case, seed):
    if case["op"] == "batch":
        qs, counts = _batch_queries(case, seed)
        return {"op": "batch", "queries": qs, "counts": counts, "batch": qbatch.Batch(qs)}
    return {"op": case["op"], "case": case, "ctx": context(), "in": _inputs(case, seed)}


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def run(state):
    op = state["op"]
    if op == "batch":
        state["batch"].run()
        state["batch"].check()
        return [q["out"] for q in state["queries"]], state["counts"]
    ctx, d = state["ctx"], state["in"]
    if op == "filter":
        return ctx.filter_cols(d["key"], d["pay"], d["lo"], d["hi"])
    if op == "filter_rec":
        return ctx.filter_range_rec(d["rec"], d["lo"], d["hi"])
    if op == "groupby":
        cap = state["case"]["groups"]
        if state["case"]["fused"]:
            return ctx.groupby_cols(d["key"], d["val"], d["val2"], d["lo2"], d["hi2"], cap=cap)
        return ctx.groupby_cols(d["key"], d["val"], cap=cap)
    if op == "groupby_ids":
        return ctx.groupby_cols(d["key"], d["val"], cap=state["case"]["groups"])
    if op == "records":
        rec, start = ctx.groupby_rec(d["rec"])
        return rec, start, ctx.aggregate_groups(rec, start, SUM)
    # room for the expected share (30 % of the probe rows) and some more
    return ctx.join_filter_sort(d["rkey"], d["rpay"], d["skey"], d["spay"], d["slo"], d["shi"],
                                cap=d["skey"].numel() // 2)


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _distinct_zipf(n, groups, share=1.0):
    """Expected distinct keys among n * share draws of the Zipf(1.0) distribution."""
    p = 1.0 / torch.arange(1, groups + 1, dtype=torch.float64)
    p /= p.sum()
    return float((-torch.expm1(n * share * torch.log1p(-p.clamp(max=1 - 1e-12)))).sum())


def _rows_bytes(op, n, nr=0, groups=0, sel=0.0):
    """Inputs read once, outputs written once."""
    if op in ("filter", "filter_rec"):
        return 8 * n + 8 * n * sel
    if op == "groupby":
        return 8 * n + 20 * _distinct_zipf(n, groups)
    if op == "fused":
        return 12 * n + 20 * _distinct_zipf(n, groups, 0.5)
    return 8 * (n + nr) + 12 * (0.8 * 0.3 * n)  # join: four fifths of the probe rows match


def work(case):
    op = case["op"]
    if op in ("filter", "filter_rec"):
        b = _rows_bytes(op, case["n"], sel=case["sel"])
    elif op == "groupby":
        b = (12 if case["fused"] else 8) * case["n"] + 20 * case["groups"]
    elif op == "groupby_ids":
        b = 8 * case["n"] + 20 * case["groups"]
    elif op == "records":
        b = 16 * case["n"] + 8 * case["groups"]
    elif op == "join":
        b = _rows_bytes("join", case["ns"], nr=case["nr"])
    elif op == "join_skew":
        b = 8 * (case["nr"] + case["ns"]) + 12 * _skew_hits(case["nr"], case["ns"])
    else:
        rng = torch.Generator().manual_seed(4 * case["each"] + 1)
        b = 0
        for i in range(4 * case["each"]):
            n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** float(torch.rand(1, generator=rng))))
            kind = {qbatch.OP_FILTER: "filter", qbatch.OP_GROUPBY: "groupby", qbatch.OP_FUSED: "fused",
                    qbatch.OP_JOIN: "join"}[i % 4]
            b += _rows_bytes(kind, n, nr=max(n // 16, 16), groups=1 << 20, sel=0.1)
    return {"bytes": b, "flops": 0}


# --------------------------------------------------------------------------
# The same results from plain torch, in 64 bits
# --------------------------------------------------------------------------
def _exact_filter(d):
    at = torch.nonzero((d["key"] >= d["lo"]) & (d["key"] <= d["hi"])).reshape(-1)
    return torch.stack([at, d["pay"][at].to(torch.int64)], dim=1)


def _exact_groupby(key, val, keep=None):
    if keep is not None:
        key, val = key[keep], val[keep]
    k, inv = torch.unique(key.to(torch.int64) & 0xFFFFFFFF, return_inverse=True)
    s = torch.zeros(k.numel(), dtype=torch.int64, device=key.device).index_add_(0, inv, val.to(torch.int64))
    c = torch.bincount(inv, minlength=k.numel())
    return torch.where(k >= 2 ** 31, k - 2 ** 32, k), s, c


def _exact_fused(d):
    return _exact_groupby(d["key"], d["val"], (d["val2"] >= d["lo2"]) & (d["val2"] <= d["hi2"]))


def _exact_join(d):
    rk, order = torch.sort(d["rkey"].to(torch.int64) & 0xFFFFFFFF)
    keep = (d["spay"] >= d["slo"]) & (d["spay"] <= d["shi"])
    sk, so = torch.sort(d["skey"][keep].to(torch.int64) & 0xFFFFFFFF)
    at = torch.searchsorted(rk, sk).clamp_(max=rk.numel() - 1)
    hit = rk[at] == sk
    sk, at = sk[hit], at[hit]
    sp = d["spay"][keep][so][hit].to(torch.int64)
    return torch.where(sk >= 2 ** 31, sk - 2 ** 32, sk), d["rpay"][order[at]].to(torch.int64), sp


def _padded(parts, like):
    out = [torch.zeros(t.shape, dtype=torch.int64, device=t.device) for t in like]
    for o, p in zip(out, parts):
        o[: p.shape[0]] = p
    return out


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        qs, counts = _batch_queries(case, seed)
        outs = []
        for i, q in enumerate(qs):
            a = q["inp"]
            if q["op"] == qbatch.OP_FILTER:
                r = (_exact_filter({"key": a[0], "pay": a[1], "lo": q["lo"], "hi": q["hi"]}),)
            elif q["op"] == qbatch.OP_GROUPBY:
                r = _exact_groupby(a[0], a[1])
            elif q["op"] == qbatch.OP_FUSED:
                r = _exact_fused({"key": a[0], "val": a[1], "val2": a[2], "lo2": q["lo"], "hi2": q["hi"]})
            else:
                r = _exact_join({"rkey": a[0], "rpay": a[1], "skey": a[2], "spay": a[3], "slo": q["lo"],
                                 "shi": q["hi"]})
            outs.append(_padded(r, q["out"]))
            counts[i] = r[0].shape[0]
        return outs, counts
    d = _inputs(case, seed)
    if op == "filter":
        return _exact_filter(d)
    if op == "filter_rec":
        return d["rec"][(d["rec"][:, 1] >= d["lo"]) & (d["rec"][:, 1] <= d["hi"])].to(torch.int64)
    if op == "groupby":
        return _exact_fused(d) if case["fused"] else _exact_groupby(d["key"], d["val"])
    if op == "groupby_ids":
        return _exact_groupby(d["key"], d["val"])
    if op == "records":
        y, order = torch.sort(d["rec"][:, 1], stable=True)
        x = d["rec"][:, 0][order].to(torch.int64)
        k, s, c = _exact_groupby(y, x)
        return torch.stack([x, y.to(torch.int64)], dim=1), torch.cumsum(c, 0) - c, s
    return _exact_join(d)
