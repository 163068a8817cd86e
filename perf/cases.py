"""The relational-operator calls whose speed this project is measured by.

Each case is one query step (or a short chain of them) over device columns,
called through ghive_b200.ops as a program does: a filter with its row count
read back, GROUP BY ... ORDER BY, a map join (build + probe), ORDER BY, and a
captured batch of group-bys.  Columns follow the shapes of
ghive_b200/workloads.py (a star schema's fact table, its dimension joins and
its sorts), generated on the device from the seed.
"""
import math

import torch

from ghive_b200 import abi, ops, workloads

DEVICE = "cuda:0"
DAYS = 2526            # days of the fact table's date column
_ctx = None


def context():
    """One context per process, as a long-running executor keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = ops.Context(0)
    return _ctx


def listed():
    return [
        # a small split's filter: launches, synchronisations and host work
        {"name": "filter_10k", "op": "filter", "rows": 10_000, "share": 0.5, "nulls": False},
        # the fact-table filter of the benchmark: d < cut, four columns out
        {"name": "filter_6m", "op": "filter", "rows": 6_000_000, "share": 0.5, "nulls": False},
        # a selective WHERE of two conditions over nullable columns, ragged size
        {"name": "filter_nulls_40m", "op": "filter", "rows": 40_000_003, "share": 0.08, "nulls": True},
        # the fact-table aggregation of the benchmark, ORDER BY its key
        {"name": "groupby_6m", "op": "groupby", "rows": 6_000_000, "groups": 1000, "key": "int",
         "theta": 0.0, "share": 0.5},
        # per-customer totals: many 64-bit keys of uneven frequency
        {"name": "groupby_wide_16m", "op": "groupby", "rows": 16_000_001, "groups": 1_000_000, "key": "long",
         "theta": 0.6, "share": 0.9},
        # GROUP BY two columns, one of them nullable, of a selective query
        {"name": "groupby_two_keys_12m", "op": "groupby2", "rows": 12_000_000, "groups": 7, "brands": 1000,
         "share": 0.3},
        # a whole-table aggregate without GROUP BY
        {"name": "aggregate_50m", "op": "aggregate", "rows": 50_000_000, "share": 0.4},
        # the benchmark's headline: dimension-table build + fact-table probe
        {"name": "join_60m", "op": "join", "build": 1_500_000, "probe": 60_000_000, "miss": 0.05},
        # LEFT OUTER on natural (spread) keys, some of them twice in the build
        {"name": "join_outer_8m", "op": "join_outer", "build": 400_000, "probe": 8_000_000, "miss": 0.1},
        # the benchmark's ORDER BY (d, k) carrying a row id
        {"name": "sort_60m", "op": "sort", "rows": 60_000_000, "zipf": False},
        # ORDER BY price DESC, region with three carried columns
        {"name": "sort_mixed_1m", "op": "sort_mixed", "rows": 1_000_000, "regions": 25},
        # many splits aggregated by one captured launch, then ordered together
        {"name": "batch_24", "op": "batch", "instances": 24, "min_rows": 10_000, "max_rows": 4_000_000},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    op = rng.choice(["filter", "groupby", "groupby2", "aggregate", "join", "join_outer", "sort", "sort_mixed",
                     "batch"])
    if op == "filter":
        return {"op": op, "rows": _log(rng, 1_000, 40_000_000), "share": round(rng.uniform(0.01, 0.95), 3),
                "nulls": rng.random() < 0.5}
    if op == "groupby":
        return {"op": op, "rows": _log(rng, 10_000, 16_000_000), "groups": _log(rng, 10, 1_000_000),
                "key": rng.choice(["int", "long"]), "theta": round(rng.uniform(0.0, 1.2), 2),
                "share": round(rng.uniform(0.05, 1.0), 3)}
    if op == "groupby2":
        return {"op": op, "rows": _log(rng, 10_000, 12_000_000), "groups": rng.randint(2, 40),
                "brands": _log(rng, 5, 4_000), "share": round(rng.uniform(0.05, 1.0), 3)}
    if op == "aggregate":
        return {"op": op, "rows": _log(rng, 10_000, 50_000_000), "share": round(rng.uniform(0.05, 1.0), 3)}
    if op == "join":
        return {"op": op, "build": _log(rng, 1_000, 1_500_000), "probe": _log(rng, 50_000, 60_000_000),
                "miss": round(rng.uniform(0.0, 0.6), 3)}
    if op == "join_outer":
        return {"op": op, "build": _log(rng, 1_000, 400_000), "probe": _log(rng, 50_000, 8_000_000),
                "miss": round(rng.uniform(0.0, 0.6), 3)}
    if op == "sort":
        return {"op": op, "rows": _log(rng, 2_000, 60_000_000), "zipf": rng.random() < 0.5}
    if op == "sort_mixed":
        return {"op": op, "rows": _log(rng, 2_000, 4_000_000), "regions": rng.randint(2, 1000)}
    return {"op": op, "instances": rng.randint(8, 32), "min_rows": 2_000,
            "max_rows": _log(rng, 100_000, 4_000_000)}


# ---------------------------------------------------------------- columns
class _Gen:
    """Device columns from one seed.  How many rows pass a filter, find a
    partner or fall into which number of groups depends on the case alone."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE)
        self.g.manual_seed(seed)

    def ints(self, lo, hi, n, dtype):
        return torch.randint(lo, hi, (n,), generator=self.g, device=DEVICE, dtype=dtype)

    def unit(self, n):
        return torch.rand(n, generator=self.g, device=DEVICE, dtype=torch.float64)

    def shuffle(self, n):
        return torch.randperm(n, generator=self.g, device=DEVICE)

    def price(self, n):
        """Money with two decimals, 900.00 to 105000.00."""
        return self.ints(90000, 10500001, n, torch.int64).to(torch.float64) / 100.0

    def days(self, n, kept, cut):
        """Dates of which the first `kept` are below `cut` and no others."""
        below = self.ints(0, cut, kept, torch.int32)
        return torch.cat([below, self.ints(min(cut, DAYS - 1), DAYS, n - kept, torch.int32)])

    def ranks(self, n, distinct, theta):
        """Ranks in [0, distinct), frequency proportional to (rank + 1) ** -theta,
        each of them at least once among the first `distinct`."""
        every = torch.arange(distinct, device=DEVICE)
        if theta <= 0.0:
            return torch.cat([every, self.ints(0, distinct, n - distinct, torch.int64)])
        cdf = torch.cumsum((every + 1).to(torch.float64).pow(-theta), 0)
        cdf /= cdf[-1].clone()
        r = torch.searchsorted(cdf, self.unit(n - distinct), right=True)
        return torch.cat([every, torch.clamp(r, max=distinct - 1)])


def _cut(case):
    return max(1, min(DAYS, int(round(case["share"] * DAYS))))


def _kept(case, n):
    """Rows that pass the date filter."""
    return n if _cut(case) == DAYS else max(1, n * _cut(case) // DAYS)


def _fact(g, keys, kept, cut):
    """The fact table's columns k, qty, price, d in random row order."""
    n = len(keys)
    at = g.shuffle(n)
    return [keys[at], g.ints(1, 51, n, torch.int64), g.price(n), g.days(n, kept, cut)[at]]


def _batch_sizes(case):
    """(rows, groups, kept, cut, theta) of each instance."""
    out, steps = [], max(1, case["instances"] - 1)
    for i in range(case["instances"]):
        n = int(case["min_rows"] * (case["max_rows"] / case["min_rows"]) ** (i / steps))
        mix = (i * 7 % case["instances"]) / steps         # sizes and shapes vary independently
        cut = int((0.05 + 0.85 * mix) * DAYS)
        kept = max(1, n * cut // DAYS)
        groups = min(kept, int(10 * 10_000 ** ((i * 5 % case["instances"]) / steps)))
        out.append((n, groups, kept, cut, 1.2 * (1 - mix)))
    return out


def _columns(case, seed):
    g, op = _Gen(seed), case["op"]
    if op == "filter":
        n = case["rows"]
        cols = _fact(g, g.ints(0, 1000, n, torch.int32), _kept(case, n), _cut(case))
        if not case["nulls"]:
            return {"cols": cols, "nulls": {}}
        # qty 1..50 and its NULLs in fixed numbers among the rows of each date class
        order = torch.argsort(cols[3] >= _cut(case), stable=True)
        i = torch.arange(n, device=DEVICE)
        cols[1][order] = 1 + i % 50
        null = torch.empty(n, dtype=torch.uint8, device=DEVICE)
        null[order] = (i // 50 % 50 == 0).to(torch.uint8)
        return {"cols": cols, "nulls": {1: null, 2: (g.unit(n) < 0.05).to(torch.uint8)}}
    if op == "groupby":
        n = case["rows"]
        kept = _kept(case, n)
        ranks = g.ranks(n, min(case["groups"], kept), case["theta"])
        return {"cols": _fact(g, ranks.to(torch.int32) if case["key"] == "int" else workloads.mix64_torch(ranks),
                              kept, _cut(case))}
    if op == "groupby2":
        n, brands = case["rows"], case["brands"]
        kept = _kept(case, n)
        pair = g.ranks(n, min(kept, case["groups"] * (brands + 1)), 0.0)    # (year, brand or NULL)
        at = g.shuffle(n)
        pair = pair[at]
        brand = pair % (brands + 1)
        return {"cols": [(1992 + pair // (brands + 1)).to(torch.int32), (brand * 10 + 1).to(torch.int32),
                         g.ints(1, 51, n, torch.int64), g.price(n), g.days(n, kept, _cut(case))[at]],
                "nulls": {1: (brand == brands).to(torch.uint8)}}
    if op == "aggregate":
        n = case["rows"]
        return {"cols": _fact(g, g.ints(0, 1000, n, torch.int32), _kept(case, n), _cut(case))}
    if op == "join":
        b, n = case["build"], case["probe"]
        fk = g.ints(1, b + 1, n, torch.int64)
        fk[:int(case["miss"] * n)] += b
        return {"bkey": g.shuffle(b) + 1, "bpay": [g.ints(0, 1 << 62, b, torch.int64), g.unit(b)],
                "fk": fk[g.shuffle(n)]}
    if op == "join_outer":
        b, n = case["build"], case["probe"]
        twice, misses = b // 10, int(case["miss"] * n)
        hits2 = (n - misses) // 10                        # probe rows of the keys that the build has twice
        rank = torch.cat([torch.arange(b, device=DEVICE), torch.arange(twice, device=DEVICE)])[g.shuffle(b + twice)]
        fk = torch.cat([g.ints(b, 2 * b, misses, torch.int64), g.ints(0, twice, hits2, torch.int64),
                        g.ints(twice, b, n - misses - hits2, torch.int64)])[g.shuffle(n)]
        mix = g.ints(1, 1 << 30, 1, torch.int64)
        return {"bkey": workloads.mix64_torch(rank + mix), "bpay": [rank * 7 + mix, (rank + mix).to(torch.float64) / 8.0],
                "fk": workloads.mix64_torch(fk + mix), "ppay": g.ints(0, 1 << 30, n, torch.int32)}
    if op == "sort":
        n = case["rows"]
        d = g.ints(0, DAYS, n, torch.int32)
        if case["zipf"]:
            vals = g.ints(0, 1 << 40, 1_000_000, torch.int64)
            w = torch.cumsum(torch.arange(1, len(vals) + 1, device=DEVICE, dtype=torch.float64).pow(-0.99), 0)
            k = vals[torch.clamp(torch.searchsorted(w / w[-1], g.unit(n), right=True), max=len(vals) - 1)]
        else:
            k = g.ints(0, 1 << 40, n, torch.int64)
        return {"keys": [d, k], "pay": [torch.arange(n, device=DEVICE, dtype=torch.int32)]}
    if op == "sort_mixed":
        n = case["rows"]
        return {"keys": [g.price(n), g.ints(0, case["regions"], n, torch.int32)],
                "nulls": (g.unit(n) < 0.03).to(torch.uint8),
                "pay": [g.ints(1, 51, n, torch.int64), torch.arange(n, device=DEVICE, dtype=torch.int32), g.unit(n)]}
    insts = []
    for n, groups, kept, cut, theta in _batch_sizes(case):
        insts.append({"cols": _fact(g, workloads.mix64_torch(g.ranks(n, groups, theta)), kept, cut),
                      "groups": groups, "cut": cut})
    return {"insts": insts}


AGGS = workloads.AGGS_FACT          # COUNT(*), SUM(qty), SUM(price), AVG(price), MIN(d), MAX(d)
AGGS2 = [(abi.CNT, -1), (abi.SUM, 2), (abi.AVG, 3), (abi.MAX, 3)]
AGGS0 = [(abi.CNT, -1), (abi.SUM, 1), (abi.SUM, 2), (abi.MIN, 2), (abi.MAX, 3)]


def _nullable(cols, nulls):
    return [(c, nulls[i]) if i in nulls else c for i, c in enumerate(cols)]


def _filter_pred(case):
    if not case["nulls"]:
        return workloads.fact_predicate(_cut(case))
    # qty BETWEEN 1 AND 40 AND d < cut, over nullable qty and price
    return abi.Pred.and_(abi.Pred.leaf(abi.FILTER_EQ_RANGE, 1, 1, 40), abi.Pred.leaf(abi.FILTER_LT, 3, a=_cut(case)))


def prepare(case, seed):
    s = _columns(case, seed)
    s["case"], s["ctx"], op = case, context(), case["op"]
    if op == "filter":
        s["in"] = _nullable(s["cols"], s["nulls"])
        s["pred"] = _filter_pred(case)
    elif op in ("groupby", "groupby2", "aggregate"):
        s["in"] = _nullable(s["cols"], s.get("nulls", {}))
        s["pred"] = abi.Pred.leaf(abi.FILTER_LT, len(s["cols"]) - 1, a=_cut(case))
    elif op == "join":
        n = case["probe"]
        # output columns a program running the query again and again keeps
        s["outs"] = (ops._Outs([abi.LONG, abi.DOUBLE], n, DEVICE, with_nulls=False), ops._Outs([], n, DEVICE),
                     torch.empty(n, dtype=torch.int32, device=DEVICE), None,
                     torch.zeros(1, dtype=torch.int64, device=DEVICE))
    elif op == "batch":
        s["batch"] = s["ctx"].batch_groupby(
            [(workloads.batched_predicate(i["cut"]), i["cols"], i["groups"], i["groups"]) for i in s["insts"]],
            [0], AGGS, autotune=False)
    return s


# ---------------------------------------------------------------- one pass
def _ordered(ctx, keys, vals, null=None):
    """ORDER BY the group keys, carrying the aggregates."""
    ks, vs, _ = ctx.sort([k if n is None else (k, n) for k, n in zip(keys, null or [None] * len(keys))],
                         payload=vals, with_nulls=False)
    return [k for k, _ in ks] + [v for v, _ in vs]


def run(s):
    case, ctx = s["case"], s["ctx"]
    op = case["op"]
    if op == "filter":
        if case["nulls"]:
            cols, _ = ctx.filter(s["pred"], s["in"], proj=[0, 2, 3])
            return [x for c in cols for x in c]
        cols, _ = ctx.filter(s["pred"], s["in"], with_nulls=False)
        return [c for c, _ in cols]
    if op == "groupby":
        ks, vs, _ = ctx.filter_groupby(s["pred"], s["in"], [0], AGGS, capacity=case["groups"],
                                       max_groups=case["groups"])
        return _ordered(ctx, [ks[0][0]], [v for v, _ in vs])
    if op == "groupby2":
        cap = case["groups"] * (case["brands"] + 1)
        ks, vs, _ = ctx.filter_groupby(s["pred"], s["in"], [0, 1], AGGS2, capacity=cap, max_groups=cap)
        return _ordered(ctx, [k for k, _ in ks], [v for v, _ in vs], [None, ks[1][1]])
    if op == "aggregate":
        _, vs, _ = ctx.filter_groupby(s["pred"], s["in"], [], AGGS0, capacity=1, max_groups=1)
        return [v for v, _ in vs]
    if op == "join":
        table = ctx.join_build(s["bkey"], build_payload=s["bpay"])
        r = ctx.join_probe(table, s["fk"], capacity=case["probe"], outs=s["outs"])
        table.free()
        return [r["probe_rowid"]] + [c for c, _ in r["build"]]
    if op == "join_outer":
        table = ctx.join_build(s["bkey"], build_payload=s["bpay"])
        r = ctx.join_probe(table, s["fk"], join_type=abi.LEFT_OUTER_JOIN, probe_payload=[s["ppay"]],
                           capacity=case["probe"] + case["probe"] // 4 + 1024, rowids=False)
        table.free()
        return [r["probe"][0][0]] + [x for c in r["build"] for x in c]
    if op == "sort":
        ks, vs, _ = ctx.sort(s["keys"], payload=s["pay"], with_nulls=False)
        return [k for k, _ in ks] + [v for v, _ in vs]
    if op == "sort_mixed":
        ks, vs, _ = ctx.sort([s["keys"][0], (s["keys"][1], s["nulls"])], orders=[abi.DESC, abi.ASC],
                             payload=s["pay"])
        return [ks[0][0], ks[1][0], ks[1][1]] + [v for v, _ in vs]
    b = s["batch"]
    b.launch()
    ctx.sync()
    counts = b.groups.tolist()
    cols = [torch.cat([b.outs[i].cols[j][0][:c] for i, c in enumerate(counts)]) for j in range(1 + len(AGGS))]
    inst = torch.repeat_interleave(torch.arange(len(counts), device=DEVICE, dtype=torch.int32), b.groups,
                                   output_size=len(cols[0]))
    return _ordered(ctx, [inst, cols[0]], cols[1:])


# ---------------------------------------------------------------- work
_WIDTH = {"int": 4, "long": 8}


def work(case):
    """Bytes of the input columns read once and of the outputs written once."""
    op = case["op"]
    flops = 0
    if op == "filter":
        n, kept = case["rows"], _kept(case, case["rows"])
        if case["nulls"]:   # k, qty, price, d and two NULL maps in; k, price, d and their NULL maps out
            b = n * 26 + 0.98 * 0.8 * kept * 19
        else:
            b = n * 24 + kept * 24
    elif op == "groupby":
        w, n = _WIDTH[case["key"]], case["rows"]
        b = n * (w + 20) + min(case["groups"], _kept(case, n)) * (w + 40)
        flops = 2 * n
    elif op == "groupby2":
        n = case["rows"]
        b = n * 29 + min(_kept(case, n), case["groups"] * (case["brands"] + 1)) * 40
        flops = 2 * n
    elif op == "aggregate":
        b = case["rows"] * 20 + 40
        flops = 3 * case["rows"]
    elif op == "join":
        b = case["build"] * 24 + case["probe"] * 8 + case["probe"] * (1 - case["miss"]) * 20
    elif op == "join_outer":
        b = case["build"] * 1.1 * 24 + case["probe"] * (12 + 22 * (1 + 0.1 * (1 - case["miss"])))
    elif op == "sort":
        b = case["rows"] * 32
    elif op == "sort_mixed":
        b = case["rows"] * (33 + 33)
    else:
        b = sum(n * 28 + groups * 48 for n, groups, _, _, _ in _batch_sizes(case))
    return {"bytes": int(b), "flops": flops}


# ---------------------------------------------------------------- exact
def _groups(key, keep, cols, aggs):
    """Aggregates per value of the int64 key of the kept rows, in key order."""
    uniq, inv = torch.unique(key[keep], return_inverse=True)
    cols = [c[keep] for c in cols]
    n, out = len(uniq), []
    count = torch.bincount(inv, minlength=n)
    for kind, c in aggs:
        if kind == abi.CNT:
            out.append(count)
        elif kind in (abi.SUM, abi.AVG):
            if cols[c].dtype == torch.float64:    # prices are whole cents: exact in int64
                cents = torch.round(cols[c] * 100.0).to(torch.int64)
                v = torch.zeros(n, dtype=torch.int64, device=DEVICE).index_add_(0, inv, cents).to(torch.float64) / 100.0
                out.append(v / count if kind == abi.AVG else v)
            else:
                out.append(torch.zeros(n, dtype=torch.int64, device=DEVICE).index_add_(0, inv, cols[c].to(torch.int64)))
        else:
            how = "amin" if kind == abi.MIN else "amax"
            out.append(torch.zeros(n, dtype=cols[c].dtype, device=DEVICE).scatter_reduce_(0, inv, cols[c], how,
                                                                                          include_self=False))
    return uniq, out


def exact(case, seed):
    s, op = _columns(case, seed), case["op"]
    if op == "filter":
        cols = s["cols"]
        keep = cols[3] < _cut(case)
        if case["nulls"]:
            keep &= (s["nulls"][1] == 0) & (cols[1] <= 40)
            none = torch.zeros(int(keep.sum()), dtype=torch.bool, device=DEVICE)
            return [cols[0][keep], none, cols[2][keep], s["nulls"][2][keep] != 0, cols[3][keep], none]
        return [c[keep] for c in cols]
    if op == "groupby":
        cols = s["cols"]
        uniq, out = _groups(cols[0].to(torch.int64), cols[3] < _cut(case), cols, AGGS)
        return [uniq.to(cols[0].dtype)] + out
    if op == "groupby2":
        cols = s["cols"]
        # NULL sorts first
        brand = torch.where(s["nulls"][1] != 0, torch.full_like(cols[1], -1), cols[1])
        key = cols[0].to(torch.int64) * (1 << 32) + brand + 1
        uniq, out = _groups(key, cols[4] < _cut(case), cols, AGGS2)
        brand = (uniq % (1 << 32)).to(torch.int32) - 1
        brand = torch.where(brand < 0, torch.full_like(brand, 2**31 - 1), brand)
        return [(uniq >> 32).to(torch.int32), brand] + out
    if op == "aggregate":
        cols = s["cols"]
        _, out = _groups(torch.zeros_like(cols[1]), cols[3] < _cut(case), cols, AGGS0)
        return out
    if op == "join":
        pos = torch.empty(2 * case["build"] + 1, dtype=torch.int64, device=DEVICE).fill_(-1)
        pos[s["bkey"]] = torch.arange(case["build"], device=DEVICE)
        at = pos[s["fk"]]
        hit = at >= 0
        return [torch.nonzero(hit).squeeze(1).to(torch.int32)] + [c[at[hit]] for c in s["bpay"]]
    if op == "join_outer":
        keys, first, = torch.unique(s["bkey"], return_inverse=True)
        times = torch.bincount(first, minlength=len(keys))
        pay = [torch.empty(len(keys), dtype=c.dtype, device=DEVICE).scatter_(0, first, c) for c in s["bpay"]]
        at = torch.clamp(torch.searchsorted(keys, s["fk"]), max=len(keys) - 1)
        miss = keys[at] != s["fk"]
        rows = torch.repeat_interleave(torch.arange(len(at), device=DEVICE), torch.where(miss, 1, times[at]))
        at, miss = at[rows], miss[rows]
        return [s["ppay"][rows], torch.where(miss, 2**63 - 1, pay[0][at]), miss,
                torch.where(miss, math.nan, pay[1][at]), miss]
    if op == "sort":
        d, k = s["keys"]
        perm = torch.sort((d.to(torch.int64) << 40) | k, stable=True).indices
        return [d[perm], k[perm], s["pay"][0][perm]]
    if op == "sort_mixed":
        price, region = s["keys"]
        null = s["nulls"] != 0
        region = torch.where(null, torch.full_like(region, 2**31 - 1), region)
        minor = torch.where(null, torch.full_like(region, -1), region)
        perm = torch.sort(minor, stable=True).indices
        perm = perm[torch.sort(price[perm], stable=True, descending=True).indices]
        return [price[perm], region[perm], null[perm]] + [c[perm] for c in s["pay"]]
    parts = []
    for i, inst in enumerate(s["insts"]):
        uniq, out = _groups(inst["cols"][0], inst["cols"][3] < inst["cut"], inst["cols"], AGGS)
        parts.append([torch.full((len(uniq),), i, dtype=torch.int32, device=DEVICE), uniq] + out)
    return [torch.cat([p[j] for p in parts]) for j in range(len(parts[0]))]
