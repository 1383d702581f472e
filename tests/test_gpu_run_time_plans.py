"""Plans without a group key that no signature covers, in the warp-tile form
against numpy: one to eight steps over columns read in every way (raw, literal
and match-bearing LZ4, packed, few-run and constant pages), every aggregate,
probes of the three table layouts, ragged tiles and parts of tiles."""
import numpy as np
import pytest

from golap_public_b200 import _lib as L
from golap_public_b200 import api

pytestmark = pytest.mark.gpu
ROWS = [1, 5, 127, 129, 1023, 1025, 40_000, 70_003, 600_001]
AGGS = {"sum": L.GX_AGG_SUM, "product": L.GX_AGG_SUM_PRODUCT, "diff": L.GX_AGG_SUM_DIFF, "count": L.GX_AGG_COUNT}


@pytest.fixture(autouse=True)
def _warp_form():
    api.set_scan_form("warp")
    yield
    api.set_scan_form("auto")


def _columns(n):
    r = np.random.default_rng(n)
    v = {"raw": r.integers(-2**31 + 1, 2**31, n), "lit": r.integers(0, 1000, n), "match": r.integers(0, 11, n),
         "pack": r.integers(-300, 3000, n), "runs": np.sort(r.integers(0, n // 700 + 2, n)),
         "const": np.full(n, 77), "inc": np.cumsum(r.integers(0, 5, n))}
    codec = {"raw": "none", "lit": "lz4", "match": "lz4"}
    kw = {"match": {"lz4_min_match": 4}}
    return v, {k: api.Column(x.astype(np.int32), codec.get(k, "cascaded"), rows_per_chunk=40_000,
                             **kw.get(k, {})).to_device() for k, x in v.items()}


@pytest.mark.parametrize("agg", list(AGGS))
@pytest.mark.parametrize("n", ROWS)
def test_random_plans(cuda, n, agg):
    v, cols = _columns(n)
    r = np.random.default_rng(n * 7 + len(agg))
    names = list(v)
    keys = {k: np.unique(x)[::2] for k, x in v.items()}
    tabs = {}
    for k, x in keys.items():
        x = x[:200_000].astype(np.int32)
        tabs[k] = (x, cuda.from_numpy(x).cuda())
    for trial in range(12):
        p = api.ScanPlan(agg=AGGS[agg], result=cuda.zeros(1, dtype=cuda.int64, device="cuda"))
        keep, carry, tables = np.ones(n, bool), None, []
        steps = int(r.integers(0, 8))
        at = int(r.integers(0, steps + 1))  # the carried column's step; the last one carries itself
        for s in range(steps + 1):
            k = str(r.choice(names))
            lo, hi = np.quantile(v[k], sorted(r.random(2) * [0.4, 0.6] + [0, 0.4])).astype(np.int64)
            if trial == 11 and s == steps // 2:
                lo, hi = 5, 4  # an empty range
            flags, ht = 0, None
            if s == steps:
                flags = L.GX_STEP_VALUE
            kind = r.integers(0, 4)
            if kind in (1, 3) or flags == 0 and kind == 0:
                flags |= L.GX_STEP_FILTER
                keep &= (v[k] >= lo) & (v[k] <= hi)
            if kind >= 2 and s < 6:
                span = int(keys[k].max()) - int(keys[k].min())
                ht = api.HashMap(len(tabs[k][0]), r.choice(["linear", "bucket", "dense"] if span < 10**6 else
                                                           ["linear", "bucket"]))
                ht.build(tabs[k][1], None)
                flags |= L.GX_STEP_PROBE
                keep &= np.isin(v[k], tabs[k][0])
                tables.append(ht)
            if s == at:
                flags |= L.GX_STEP_CARRY
                carry = v[k]
            if not flags:
                flags = L.GX_STEP_FILTER
                keep &= (v[k] >= lo) & (v[k] <= hi)
            p.steps.append(api.Step(cols[k], flags, int(lo), int(hi), ht))
        x, c = v[k][keep].astype(np.int64), carry[keep].astype(np.int64)
        with np.errstate(over="ignore"):
            want = {"sum": x.sum(), "product": (x * c).sum(), "diff": (x - c).sum(), "count": keep.sum()}[agg]
        p.launch()
        api.scan_check()
        assert int(p.result.item()) == int(want), (trial, [(st.flags, st.lo, st.hi) for st in p.steps])
