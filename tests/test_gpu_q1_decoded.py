"""The Q1 signature over columns that the warp decodes first: LZ4 with one lane
per segment (padded rows) and groups of lanes, cascaded pages of short runs,
beside direct, constant and packed ones; whole and ragged tiles."""
import numpy as np
import pytest

from golap_public_b200 import _lib as L
from golap_public_b200 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _warp_form():
    api.set_scan_form("warp")
    yield
    api.set_scan_form("auto")


def _columns(n):
    r = np.random.default_rng(n)
    runs = lambda k, hi: np.repeat(r.integers(0, hi, n // k + 1), k)[:n]
    v = {"lane": r.integers(0, 11, n), "groups": runs(30, 11), "long": runs(9, 11), "casc": runs(6, 11),
         "direct": r.integers(0, 11, n), "packed": r.integers(0, 11, n), "const": np.full(n, 5)}
    kw = {"lane": {"lz4_min_match": 4}, "groups": {"lz4_min_match": 4, "lz4_segments": 32},
          "long": {"lz4_min_match": 8, "lz4_segments": 16}}
    codec = {"casc": "cascaded", "packed": "cascaded", "const": "cascaded", "direct": "none"}
    return v, {k: api.Column(x.astype(np.int32), codec.get(k, "lz4"), rows_per_chunk=100_000,
                             **kw.get(k, {})).to_device() for k, x in v.items()}


@pytest.mark.parametrize("layout", ["linear", "dense"])
@pytest.mark.parametrize("n", [3, 1023, 1024, 1280, 70_003, 400_000])
def test_q1_over_decoded_columns(cuda, n, layout):
    v, cols = _columns(n)
    r = np.random.default_rng(n + 1)
    date = np.sort(r.integers(0, n // 500 + 3, n))
    price = r.integers(0, 2**31, n)
    mk = lambda x, c: api.Column(x.astype(np.int32), c, rows_per_chunk=100_000).to_device()
    cd, cp = mk(date, "cascaded"), mk(price, "lz4")
    days = np.unique(date)[::2].astype(np.int32)
    kd = cuda.from_numpy(days).cuda()
    ht = api.HashMap(len(days), layout).build(kd, None)
    ok = np.isin(date, days)
    res = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    for a in v:
        for b in v:
            res.zero_()
            p = api.ScanPlan(agg=L.GX_AGG_SUM_PRODUCT, result=res)
            p.probe(cd, ht).filter(cols[a], 3, 7, carry=True).filter(cols[b], 2, 8).value(cp).launch()
            api.scan_check()
            m = ok & (v[a] >= 3) & (v[a] <= 7) & (v[b] >= 2) & (v[b] <= 8)
            assert int(res.item()) == int((v[a][m] * price[m]).sum()), (a, b)
