"""The work a user of this engine has it do, as cases that can be timed.

Every case goes through the public entry points (queries.py, api.py) the way
a program calls them: the dimension tables are rebuilt and the scan launched,
a batch graph is replayed, a column is ingested or decompressed, a join or a
group-by runs on device columns.  Data are seeded and synthetic with the
distributions of datagen.py (date keys of 2,556 days, quantity U[1,50],
discount U[0,10], prices, surrogate keys 1..N, bounded Zipf part keys),
generated on the GPU so that preparing a case is quick.

A case is a dict of plain values; "kind" selects what runs:

  q1      SUM(extended_price * discount) over fact JOIN date; the date table
          is rebuilt from the predicate and the scan launched, directly or as
          a captured CUDA graph
  star    Q3: customer table built from compressed customer columns, supplier
          and date tables, three probes, GROUP BY nations and year, groups read
  profit  Q4: four probes, SUM(revenue - supplycost) GROUP BY nation and year
  group   SUM(revenue) GROUP BY part key (Zipf) over a date range; the group
          table is consumed on the device
  batch   many queries of the scan / star / group-by mix on slices of one
          table, one graph replay
  decode  a whole column decompressed into a device buffer
  ingest  the four Q1 columns encoded on the GPU, then decompressed
  join    a join table built from device columns and probed
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from golap_public_b200 import _lib as L
from golap_public_b200 import datagen, queries, workload
from golap_public_b200.api import Batch, ChunkDecompressor, Column, HashAggregate, HashMap, ScanPlan

DATE = datagen.date_dim()
DISC, QTY = (4, 6), (26, 35)  # the discount and quantity bands of Q1.2
REGION = 2
YEARS = (1992, 1997)
PARTS = 1_400_000
# compressed bytes per row, side index included, of the columns as datagen.py draws them
LZ4_LITERAL, LZ4_MATCH = 4.15, {"discount": 2.4, "quantity": 3.44, "extended_price": 4.15}
CASC = {"date_key": 2.04, "discount": 0.54, "quantity": 0.79, "extended_price": 3.04}


def listed():
    return [
        # the smallest call: a scale-factor-1 table, uncompressed and unsorted, one year, launched directly
        {"name": "q1_raw_6M_year", "kind": "q1", "rows": 6_000_000, "sorted": False, "codec": "none", "match": 0,
         "range": "year", "mode": "call"},
        # the headline query: one month of a date-sorted table; pruning leaves about 1 % of it (latency)
        {"name": "q1_month_60M_graph", "kind": "q1", "rows": 60_000_000, "sorted": True, "codec": "lz4", "match": 0,
         "range": "month", "mode": "graph"},
        # the same table with every row needed (bandwidth)
        {"name": "q1_full_60M", "kind": "q1", "rows": 60_000_000, "sorted": True, "codec": "lz4", "match": 0,
         "range": "all", "mode": "call"},
        # columns whose LZ4 blocks hold short matches, as a size-first encoder writes them; an odd row count
        {"name": "q1_full_10M_matches", "kind": "q1", "rows": 10_000_123, "sorted": True, "codec": "lz4", "match": 4,
         "range": "all", "mode": "call"},
        # every column bit-packed (cascaded), dates in arrival order: each page has to be unpacked
        {"name": "q1_full_16M_cascaded", "kind": "q1", "rows": 16_000_001, "sorted": False, "codec": "cascaded",
         "match": 0, "range": "all", "mode": "call"},
        # the large star join with its dimension tables, customer built from compressed columns
        {"name": "star_200M_dense", "kind": "star", "rows": 200_000_000, "customers": 3_000_000, "layout": "dense"},
        # the widest plan: six columns, four hashed join tables of the default layout
        {"name": "profit_24M_linear", "kind": "profit", "rows": 24_000_000, "customers": 900_000, "layout": "linear"},
        # skewed group-by with as many groups as a part dimension has keys
        {"name": "group_30M_zipf", "kind": "group", "rows": 30_000_000, "keys": PARTS},
        # concurrent users: uneven queries of all three templates over one resident table
        {"name": "batch_32_of_16M", "kind": "batch", "rows": 16_000_000, "queries": 32},
        # a column handed decompressed to other kernels
        {"name": "decode_24M_matches", "kind": "decode", "rows": 24_000_321, "codec": "lz4", "match": 4,
         "column": "discount"},
        # new data arriving in device memory
        {"name": "ingest_16M", "kind": "ingest", "rows": 16_000_000},
        # join operators on plain device columns: 1M build rows, 16M probes
        {"name": "join_1M_16M_linear", "kind": "join", "build": 1_000_000, "probe": 16_000_000, "layout": "linear"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["q1", "q1", "q1", "star", "profit", "group", "batch", "decode", "ingest", "join"])
    if kind == "q1":
        codec = rng.choice(["lz4", "lz4", "cascaded", "none"])
        match = rng.choice([0, 0, 4, 8]) if codec == "lz4" else 0
        return {"kind": kind, "rows": _log(rng, 200_000, 12_000_000 if match else 60_000_000),
                "sorted": rng.random() < 0.7, "codec": codec, "match": match,
                "range": rng.choice(["month", "year", "all"]), "mode": rng.choice(["call", "graph"])}
    if kind == "star":
        return {"kind": kind, "rows": _log(rng, 2_000_000, 120_000_000), "customers": _log(rng, 30_000, 3_000_000),
                "layout": rng.choice(["linear", "bucket", "dense"])}
    if kind == "profit":
        return {"kind": kind, "rows": _log(rng, 1_000_000, 24_000_000), "customers": _log(rng, 30_000, 3_000_000),
                "layout": rng.choice(["linear", "bucket", "dense"])}
    if kind == "group":
        return {"kind": kind, "rows": _log(rng, 500_000, 30_000_000), "keys": _log(rng, 1_000, PARTS)}
    if kind == "batch":
        return {"kind": kind, "rows": _log(rng, 2_000_000, 16_000_000), "queries": rng.randint(4, 48)}
    if kind == "decode":
        codec = rng.choice(["lz4", "lz4", "cascaded", "none"])
        return {"kind": kind, "rows": _log(rng, 100_000, 32_000_000), "codec": codec,
                "match": rng.choice([0, 4, 8]) if codec == "lz4" else 0,
                "column": rng.choice(["date_key", "discount", "quantity", "extended_price"])}
    if kind == "ingest":
        return {"kind": kind, "rows": _log(rng, 500_000, 32_000_000)}
    return {"kind": kind, "build": _log(rng, 2_000, 3_000_000), "probe": _log(rng, 100_000, 32_000_000),
            "layout": rng.choice(["linear", "bucket", "dense"])}


# ------------------------------------------------------------------ data

def _gen(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + stream) & 0x7FFFFFFFFFFFFFFF)
    return g


def _uniform(seed, stream, n, lo, hi):
    """int32 values uniform in [lo, hi)."""
    return torch.randint(lo, hi, (n,), generator=_gen(seed, stream), device="cuda", dtype=torch.int32)


def _dates(seed, n, sorted_):
    keys = torch.from_numpy(DATE["d_key"]).cuda()
    day = _uniform(seed, 1, n, 0, datagen.N_DAYS)
    if not sorted_:
        return keys[day]
    return torch.repeat_interleave(keys, torch.bincount(day, minlength=datagen.N_DAYS), output_size=n)


def _zipf(seed, n, n_keys):
    w = torch.arange(1, n_keys + 1, dtype=torch.float64, device="cuda") ** -1.1
    cdf = torch.cumsum(w, 0)
    u = torch.rand(n, generator=_gen(seed, 31), device="cuda", dtype=torch.float64) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=n_keys - 1).add_(1).to(torch.int32)


def _q1_columns(seed, n, sorted_):
    return {"date_key": _dates(seed, n, sorted_), "quantity": _uniform(seed, 2, n, 1, 51),
            "discount": _uniform(seed, 3, n, 0, 11), "extended_price": _uniform(seed, 4, n, 90_000, 10_494_951)}


def _fact_columns(seed, n, customers, suppliers, parts=PARTS):
    return {"date_key": _dates(seed, n, True), "cust_key": _uniform(seed, 12, n, 1, customers + 1),
            "supp_key": _uniform(seed, 13, n, 1, suppliers + 1), "part_key": _uniform(seed, 14, n, 1, parts + 1),
            "revenue": _uniform(seed, 15, n, 100, 1_000_001), "supplycost": _uniform(seed, 16, n, 100, 600_001)}


def _suppliers(customers):
    return max(2_000, customers // 15)


def _geo(seed, n, stream):
    """Customer or supplier dimension on the host: key, nation, region."""
    nation = _uniform(seed, stream, n, 0, 25).cpu().numpy()
    return {"key": np.arange(1, n + 1, dtype=np.int32), "nation": nation, "region": datagen.NATION_REGION[nation]}


def _part(seed, n):
    cat = _uniform(seed, 23, n, 0, 25).cpu().numpy()
    return {"key": np.arange(1, n + 1, dtype=np.int32), "category": cat, "mfgr": (cat // 5).astype(np.int32),
            "brand": (40 * cat).astype(np.int32)}


def _host(cols):
    return {k: v.cpu().numpy() for k, v in cols.items()}


def _on_gpu(cols):
    """A fact table encoded from device columns: date_key cascaded, the others LZ4 literal runs."""
    n = next(iter(cols.values())).numel()
    return queries.FactTable({k: Column.from_device(v, "cascaded" if k == "date_key" else "lz4", name=k)
                              for k, v in cols.items()}, n)


def _date_range(case):
    """(rows of the date dimension that pass, lowest key, highest key)."""
    if case["range"] == "month":
        return DATE["d_yearmonthnum"] == 199401, 19940101, 19940131
    if case["range"] == "year":
        return DATE["d_year"] == 1993, 19930101, 19931231
    return np.ones(len(DATE["d_key"]), bool), int(DATE["d_key"].min()), int(DATE["d_key"].max())


# ------------------------------------------------- grouped results on the device

class _Words:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i8", "data": (ptr, False), "version": 2}


def _group_view(agg):
    """The group table's keys and sums as device tensors (gx_groupby_view: negative key = free)."""
    k, s, log2 = C.c_void_p(), C.c_void_p(), C.c_uint32()
    L.check(L.lib().gx_groupby_view(agg.handle, C.byref(k), C.byref(s), C.byref(log2)))
    n = 1 << log2.value
    return torch.as_tensor(_Words(k.value, n), device="cuda"), torch.as_tensor(_Words(s.value, n), device="cuda")


def _dense(view, out):
    """The groups as one dense array over the key space (its last element takes the free slots)."""
    keys, sums = view
    out.zero_()
    out.scatter_(0, torch.where(keys >= 0, keys, out.numel() - 1), sums)
    return out[:-1]


# --------------------------------------------------------------- prepare

def _prepare_q1(case, seed):
    cols = _q1_columns(seed, case["rows"], case["sorted"])
    if case["codec"] == "lz4":
        codecs = {k: "lz4" for k in cols}
        codecs["date_key"] = "cascaded"
    else:
        codecs = {k: case["codec"] for k in cols}
    fact = queries.encode_fact(_host(cols), codecs, lz4_min_match=case["match"])
    ok, lo, hi = _date_range(case)
    q = queries.Q1Query(fact, DATE, ok, lo, hi, *DISC, *QTY, prune=case["range"] != "all")
    st = {"q": q, "fact": fact, "graph": None}
    if case["mode"] == "graph":
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _q1_step(q)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            _q1_step(q)
    return st


def _q1_step(q):
    q.result.zero_()
    q.ht.build(q._dk, None, preds=[(q._ok, 1, 1)])
    q.plan.launch()


def _prepare_star(case, seed):
    n_c = case["customers"]
    cols = _fact_columns(seed, case["rows"], n_c, _suppliers(n_c))
    fact = _on_gpu({k: cols.pop(k) for k in ("date_key", "cust_key", "supp_key", "revenue")})
    cust = queries.encode_fact(_geo(seed, n_c, 21), {"key": "cascaded", "nation": "cascaded", "region": "cascaded"})
    q = queries.Q3Query(fact, cust, _geo(seed, _suppliers(n_c), 22), DATE, REGION, *YEARS, ht_layout=case["layout"])
    return {"q": q, "cust": cust}


def _prepare_profit(case, seed):
    n_c = case["customers"]
    n_p = min(PARTS, max(20_000, n_c // 2))
    cols = _fact_columns(seed, case["rows"], n_c, _suppliers(n_c), n_p)
    fact = _on_gpu(cols)
    q = queries.Q4Query(fact, _geo(seed, n_c, 21), _geo(seed, _suppliers(n_c), 22), _part(seed, n_p), DATE, 1, 0, 1,
                        ht_layout=case["layout"])
    return {"q": q}


def _prepare_group(case, seed):
    n = case["rows"]
    fact = _on_gpu({"date_key": _dates(seed, n, True), "part_key": _zipf(seed, n, case["keys"]),
                    "revenue": _uniform(seed, 15, n, 100, 1_000_001)})
    agg = HashAggregate(case["keys"])
    lo, hi = YEARS[0] * 10000 + 101, YEARS[1] * 10000 + 1231
    plan = ScanPlan(agg=L.GX_AGG_SUM, groupby=agg).prune_minmax(fact.cols["date_key"], lo, hi)
    plan.filter(fact.cols["date_key"], lo, hi).group(fact.cols["part_key"], 1, case["keys"])
    plan.value(fact.cols["revenue"])
    return {"fact": fact, "agg": agg, "plan": plan, "view": _group_view(agg),
            "out": torch.empty(case["keys"] + 1, dtype=torch.int64, device="cuda")}


def _batch_table(case, seed):
    n, n_c, n_s = case["rows"], 600_000, 40_000
    cols = _q1_columns(seed, n, True)
    cols.update({"cust_key": _uniform(seed, 12, n, 1, n_c + 1), "supp_key": _uniform(seed, 13, n, 1, n_s + 1),
                 "revenue": _uniform(seed, 15, n, 100, 1_000_001), "part_key": _zipf(seed, n, PARTS)})
    return cols, _geo(seed, n_c, 21), _geo(seed, n_s, 22)


def _batch_specs(t, case):
    """The case's queries (templates, slices, parameters): the same for every seed, over other data."""
    return workload.random_queries(t, case["queries"], np.random.default_rng(case["queries"]), min_rows=1_000_000,
                                   ht_layout="linear")


def _prepare_batch(case, seed):
    cols, cust, supp = _batch_table(case, seed)
    t = workload.WideTable(case["rows"], {}, _on_gpu(cols).cols, {"customer": cust, "supplier": supp, "date": DATE})
    dk, dy = torch.from_numpy(DATE["d_key"]).cuda(), torch.from_numpy(DATE["d_year"]).cuda()
    hts = {"date": HashMap(len(DATE["d_key"])).build(dk, dy), "cust": [], "supp": []}
    for name, d in (("cust", cust), ("supp", supp)):
        k, nat, reg = (torch.from_numpy(np.ascontiguousarray(d[c])).cuda() for c in ("key", "nation", "region"))
        t._keep += [k, nat, reg]
        for r in range(5):
            hts[name].append(HashMap(max(1, int((d["region"] == r).sum()))).build(k, nat, preds=[(reg, r, r)]))
    t._keep += [dk, dy]
    t.ht["linear"] = hts
    specs = _batch_specs(t, case)
    grouped = []
    for s in specs:
        if s.groups is not None:
            y = s.params["years"]
            card = 625 * (y[1] - y[0] + 1) if s.template == "star" else PARTS
            grouped.append((_group_view(s.groups), torch.empty(card + 1, dtype=torch.int64, device="cuda")))
    batch = Batch([(s.plan, s.row_lo, s.row_hi) for s in specs])
    return {"table": t, "specs": specs, "batch": batch, "grouped": grouped,
            "scalars": [s.result for s in specs if s.groups is None]}


def _prepare_decode(case, seed):
    v = _q1_columns(seed, case["rows"], True)[case["column"]]
    col = Column(v.cpu().numpy(), case["codec"], lz4_min_match=case["match"]).to_device()
    return {"dec": ChunkDecompressor(col), "n": col.info.n_chunks, "out": torch.empty_like(v)}


def _prepare_ingest(case, seed):
    cols = _q1_columns(seed, case["rows"], True)
    return {"cols": cols, "out": {k: torch.empty_like(v) for k, v in cols.items()}}


def _join_columns(case, seed):
    """Build side: every key 1..n once, shuffled, with a payload and a region to filter on; probe keys reach
    a quarter past the build keys."""
    n = case["build"]
    key = torch.randperm(n, generator=_gen(seed, 41), device="cuda").to(torch.int32).add_(1)
    return {"key": key, "pay": _uniform(seed, 42, n, 0, 1_000_000), "reg": _uniform(seed, 43, n, 0, 5),
            "probe": _uniform(seed, 44, case["probe"], 1, n + n // 4 + 2)}


def _prepare_join(case, seed):
    st = _join_columns(case, seed)
    st["ht"] = HashMap(case["build"], case["layout"])
    st["out"] = torch.empty_like(st["probe"])
    st["hits"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    return st


def prepare(case, seed):
    st = globals()["_prepare_" + case["kind"]](case, seed)
    st["kind"] = case["kind"]
    return st


# ------------------------------------------------------------------- run

def _rows(groups, width):
    """{key tuple: sum} as int64 arrays ordered by key."""
    items = sorted(groups.items())
    return {"keys": np.array([k for k, _ in items], np.int64).reshape(-1, width),
            "sums": np.array([v for _, v in items], np.int64)}


def run(state):
    kind = state["kind"]
    if kind == "q1":
        q = state["q"]
        if state["graph"] is not None:
            state["graph"].replay()
        else:
            _q1_step(q)
        return {"sum": q.result, "keep": q.keep}
    if kind == "star":
        q = state["q"]
        q.build_customer()
        sk, sn, sr, dk, dy = q._keep_alive[3:8]
        q.hs.build(sk, sn, preds=[(sr, REGION, REGION)])
        q.hd.build(dk, dy, preds=[(dy, *YEARS)])
        return _rows(q.run(), 3)
    if kind == "profit":
        return _rows(state["q"].run(), 2)
    if kind == "group":
        state["agg"].reset()
        state["plan"].launch()
        return _dense(state["view"], state["out"])
    if kind == "batch":
        state["batch"].graph()
        return {"sums": state["scalars"], "groups": [_dense(v, o) for v, o in state["grouped"]]}
    if kind == "decode":
        state["dec"].chunks(0, state["n"], state["out"])
        return state["out"]
    if kind == "ingest":
        got = {}
        for name, v in state["cols"].items():
            col = Column.from_device(v, "cascaded" if name == "date_key" else "lz4", name=name)
            ChunkDecompressor(col).chunks(0, col.info.n_chunks, state["out"][name])
            got[name] = {"rows": state["out"][name], "minmax": col.minmax(), "blocks": col.block_minmax(),
                         "bytes": col.info.comp_bytes}
        return got
    state["ht"].build(state["key"], state["pay"], preds=[(state["reg"], 0, 2)])
    state["hits"].zero_()
    state["ht"].probe(state["probe"], state["out"], state["hits"])
    return {"payload": state["out"], "hits": state["hits"]}


# ------------------------------------------------------------------ work

def work(case):
    """Compressed bytes of the rows the query has to look at, plus what it writes."""
    kind, n = case["kind"], case.get("rows", 0)
    if kind == "q1":
        part = {"month": 31 / datagen.N_DAYS, "year": 365 / datagen.N_DAYS, "all": 1.0}[case["range"]]
        if case["codec"] == "none":
            row = 16.0
        elif case["codec"] == "cascaded":
            row = sum(CASC.values()) - (CASC["date_key"] if case["sorted"] else 0)
        else:
            row = sum(LZ4_MATCH.values()) if case["match"] else 3 * LZ4_LITERAL
            row += 0 if case["sorted"] else CASC["date_key"]
        if not case["sorted"]:
            part = 1.0
        return {"bytes": n * row * part + 12 * len(DATE["d_key"]), "flops": 0}
    if kind == "star":
        c, s = case["customers"], _suppliers(case["customers"])
        return {"bytes": 3 * LZ4_LITERAL * n * 6 / 7 + 2.5 * c + 12 * s + 8 * (c + s) / 5, "flops": 0}
    if kind == "profit":
        return {"bytes": 5 * LZ4_LITERAL * n, "flops": 0}
    if kind == "group":
        return {"bytes": 2 * LZ4_LITERAL * n * 6 / 7 + 16 * case["keys"], "flops": 0}
    if kind == "batch":
        return {"bytes": 7 * LZ4_LITERAL * n, "flops": 0}
    if kind == "decode":
        comp = 4.15
        if case["codec"] == "cascaded":
            comp = 0.03 if case["column"] == "date_key" else CASC[case["column"]]
        elif case["codec"] == "lz4":
            comp = 0.15 if case["column"] == "date_key" else LZ4_MATCH[case["column"]] if case["match"] else 4.15
        return {"bytes": n * (4 + comp), "flops": 0}
    if kind == "ingest":
        return {"bytes": n * (16 + 3 * LZ4_LITERAL + 16), "flops": 0}
    return {"bytes": 12 * case["build"] + 8 * 0.6 * case["build"] + 8 * case["probe"], "flops": 0}


# ----------------------------------------------------------------- exact

def _in(v, lo, hi):
    return (v >= lo) & (v <= hi)


def _sums(key, val, card):
    return torch.zeros(card, dtype=torch.int64, device="cuda").index_add_(0, key.long(), val.long())


def _table(total, seen, digits):
    """Sums of the groups seen, with their keys split into digits (base, cardinality)."""
    k = torch.nonzero(seen).flatten()
    out, r = [], k
    for base, card in reversed(digits):
        out.append(r % card + base)
        r = r // card
    return {"keys": torch.stack(out[::-1], 1), "sums": total[k]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "q1":
        c = _q1_columns(seed, case["rows"], case["sorted"])
        ok, _, _ = _date_range(case)
        good = torch.zeros(20_000_000, dtype=torch.bool, device="cuda")
        good[torch.from_numpy(DATE["d_key"][ok]).cuda().long()] = True
        m = good[c["date_key"].long()] & _in(c["discount"], *DISC) & _in(c["quantity"], *QTY)
        return {"sum": (c["extended_price"][m].long() * c["discount"][m].long()).sum().reshape(1), "keep": None}
    if kind in ("star", "profit"):
        n_c = case["customers"]
        region = REGION if kind == "star" else 1
        n_p = PARTS if kind == "star" else min(PARTS, max(20_000, n_c // 2))
        c = _fact_columns(seed, case["rows"], n_c, _suppliers(n_c), n_p)
        geo = [{k: torch.from_numpy(v).cuda() for k, v in g.items()}
               for g in (_geo(seed, n_c, 21), _geo(seed, _suppliers(n_c), 22))]
        year = c["date_key"] // 10000
        m = (geo[0]["region"] == region)[c["cust_key"].long() - 1] & (geo[1]["region"] == region)[c["supp_key"].long() - 1]
        if kind == "star":
            m &= _in(year, *YEARS)
        else:
            m &= _in(torch.from_numpy(_part(seed, n_p)["mfgr"]).cuda(), 0, 1)[c["part_key"].long() - 1]
        c = {k: v[m] for k, v in c.items()}
        year = year[m].long() - 1992
        cn = geo[0]["nation"][c["cust_key"].long() - 1].long()
        if kind == "star":
            key = (cn * 25 + geo[1]["nation"][c["supp_key"].long() - 1].long()) * 6 + year
            digits, val = [(0, 25), (0, 25), (1992, 6)], c["revenue"]
        else:
            key, digits, val = cn * 7 + year, [(0, 25), (1992, 7)], c["revenue"].long() - c["supplycost"].long()
        card = math.prod(d[1] for d in digits)
        return _table(_sums(key, val, card), _sums(key, torch.ones_like(key), card) > 0, digits)
    if kind == "group":
        n = case["rows"]
        m = _in(_dates(seed, n, True), YEARS[0] * 10000 + 101, YEARS[1] * 10000 + 1231)
        return _sums(_zipf(seed, n, case["keys"])[m] - 1, _uniform(seed, 15, n, 100, 1_000_001)[m], case["keys"])
    if kind == "decode":
        return _q1_columns(seed, case["rows"], True)[case["column"]]
    if kind == "join":
        c = _join_columns(case, seed)
        pay = torch.full((2 * case["build"] + 4,), -2 ** 31, dtype=torch.int64, device="cuda")  # -2^31: no match
        m = _in(c["reg"], 0, 2)
        pay[c["key"][m].long()] = c["pay"][m].long()
        out = pay[c["probe"].long()]
        return {"payload": out, "hits": (out != -2 ** 31).sum().reshape(1)}
    return None  # batch, ingest: whole numbers, compared as they are
