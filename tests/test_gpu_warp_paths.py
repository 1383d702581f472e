"""The warp-tile scan's read paths at their edges, against numpy on the same
columns: bit-packed pages of every word-straddling width, pages of a few runs
(more than two on a tile), ragged tiles, chains of nearly full join tables, and
group keys that overflow the CTA's table."""
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


def _col(v, codec, **kw):
    return api.Column(v.astype(np.int32), codec, rows_per_chunk=40_000, **kw).to_device()


def _sum(torch, filt, lo, hi, value, carry=None):
    res = torch.zeros(1, dtype=torch.int64, device="cuda")
    p = api.ScanPlan(agg=L.GX_AGG_SUM_PRODUCT if carry is not None else L.GX_AGG_SUM, result=res)
    p.filter(filt, lo, hi)
    if carry is not None:
        p.carry(carry)
    p.value(value)
    p.launch()
    api.scan_check()
    return int(res.item())


@pytest.mark.parametrize("bits", [1, 2, 7, 8, 9, 15, 16, 17, 24, 25, 31, 32])
@pytest.mark.parametrize("n", [1, 3, 1023, 1025, 2049, 40_001, 100_003])
def test_packed_widths(cuda, bits, n):
    r = np.random.default_rng(bits * 1000 + n)
    lo = -(1 << (bits - 1))
    v = r.integers(lo, lo + (1 << bits), n, dtype=np.int64)
    w = r.integers(0, 1000, n)
    cv, cw = _col(v, "cascaded"), _col(w, "none")
    a, b = np.quantile(v, [0.2, 0.8]).astype(np.int64)
    m = (v >= a) & (v <= b)
    assert _sum(cuda, cv, int(a), int(b), cw) == int(w[m].sum())
    assert _sum(cuda, cw, 100, 800, cv) == int(v[(w >= 100) & (w <= 800)].sum())


@pytest.mark.parametrize("run", [300, 700, 1500])
@pytest.mark.parametrize("step", [1, 1000])
def test_few_runs(cuda, run, step):
    n = 90_011
    r = np.random.default_rng(run)
    v = np.repeat(np.arange(n // run + 1) * step - 5, run)[:n]
    w, x = r.integers(-500, 500, n), r.integers(0, 50, n)
    for codec in ("cascaded", "lz4"):
        cv, cw, cx = _col(v, "cascaded"), _col(w, codec), _col(x, codec)
        a, b = int(v[n // 5]), int(v[n // 2])
        m = (v >= a) & (v <= b)
        assert _sum(cuda, cv, a, b, cw, cx) == int((w[m] * x[m]).sum())


@pytest.mark.parametrize("layout", ["linear", "bucket", "dense"])
@pytest.mark.parametrize("entries,cap", [(5, 5), (1000, 513), (4095, 2048)])
def test_chains_and_group_overflow(cuda, layout, entries, cap):
    # tables filled past their nominal load (long chains), probed with keys half
    # of which are absent; up to 4095 groups for 512 shared slots; negative values
    n = 120_007
    r = np.random.default_rng(entries)
    keys = np.arange(1, entries + 1, dtype=np.int32) * 3
    pay = r.permutation(entries).astype(np.int32)
    ht = api.HashMap(cap, layout)
    kd, pd = cuda.from_numpy(keys).cuda(), cuda.from_numpy(pay).cuda()
    ht.build(kd, pd)
    k = r.integers(0, entries + 2, n) * 3 - r.integers(0, 2, n)
    val = r.integers(-2_000_000_000, 2_000_000_000, n)
    date = np.sort(r.integers(0, 4, n))
    fact = {c: _col(x, "cascaded" if c == "d" else "lz4") for c, x in (("k", k), ("v", val), ("d", date))}
    agg = api.HashAggregate(entries * 4)
    p = api.ScanPlan(agg=L.GX_AGG_SUM, groupby=agg)
    p.probe(fact["k"], ht, 0, entries).group(fact["d"], 0, 4).value(fact["v"])
    p.launch()
    api.scan_check()
    look = np.full(entries * 3 + 10, -1, np.int64)
    look[keys] = pay
    d = look[np.maximum(k, 0)]
    d[k < 0] = -1
    m = d >= 0
    want = np.zeros(entries * 4, np.int64)
    np.add.at(want, d[m] * 4 + date[m], val[m])
    seen = np.unique(d[m] * 4 + date[m])
    assert agg.read() == {int(g): int(want[g]) for g in seen}


@pytest.mark.parametrize("n", [1, 1025, 300_001])
@pytest.mark.parametrize("date", ["sorted", "few_runs", "random"])
def test_group_by_of_a_range(cuda, n, date):
    # the group-by template (filter, group column, value): constant, two-run,
    # decoded and packed filter columns, an empty range, a digit out of range
    r = np.random.default_rng(n)
    d = {"sorted": np.sort(r.integers(0, 20, n)), "few_runs": np.sort(r.integers(0, n // 300 + 1, n)),
         "random": r.integers(0, 1000, n)}[date]
    k, v = r.integers(7, 2007, n), r.integers(-10**9, 10**9, n)
    cd, ck, cv = _col(d, "cascaded"), _col(k, "lz4"), _col(v, "none")
    for lo, hi in ((int(np.quantile(d, 0.1)), int(np.quantile(d, 0.9))), (5, 4)):
        agg = api.HashAggregate(2000)
        api.ScanPlan(agg=L.GX_AGG_SUM, groupby=agg).filter(cd, lo, hi).group(ck, 7, 2000).value(cv).launch()
        api.scan_check()
        m = (d >= lo) & (d <= hi)
        want = np.zeros(2000, np.int64)
        np.add.at(want, k[m] - 7, v[m])
        assert agg.read() == {int(g): int(want[g]) for g in np.unique(k[m] - 7)}
    agg = api.HashAggregate(2000)
    api.ScanPlan(agg=L.GX_AGG_SUM, groupby=agg).filter(cd, 0, 10**6).group(ck, 8, 2000).value(cv).launch()
    if (k == 7).any():
        with pytest.raises(api.L.GxError):
            api.scan_check()
    else:
        api.scan_check()


@pytest.mark.parametrize("rpb,S", [(4096, 128), (8192, 128), (16384, 128), (16384, 32)])
@pytest.mark.parametrize("n", [31, 1025, 70_003])
def test_short_sequences(cuda, rpb, S, n):
    # LZ4 segments of 32, 64, 128 and 512 rows full of short matches: one to
    # three such columns beside a literal one, with literal runs longer than one
    # and two extension bytes, and matches longer than a token's nibble
    r = np.random.default_rng(n + S)
    kw = dict(rows_per_block=rpb, lz4_segments=S, lz4_min_match=4)
    few = r.integers(0, 5, n)
    mixed = np.where(r.integers(0, 400, n) < 3, r.integers(-2**31, 2**31, n), r.integers(0, 9, n))
    bursts = r.integers(0, 2**31, n)
    bursts[(np.arange(n) // 40) % 3 != 0] = 7
    cols = [_col(x, "lz4", **kw) for x in (few, mixed, bursts)]
    price = r.integers(0, 2**31, n)
    cp = _col(price, "lz4", rows_per_block=rpb, lz4_segments=S)
    m = (few >= 1) & (few <= 3)
    assert _sum(cuda, cols[0], 1, 3, cp) == int(price[m].sum())
    assert _sum(cuda, cols[0], 1, 3, cols[1]) == int(mixed[m].sum())
    m &= (mixed >= 2) & (mixed <= 6)
    res = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    p = api.ScanPlan(agg=L.GX_AGG_SUM_PRODUCT, result=res)
    p.filter(cols[0], 1, 3, carry=True).filter(cols[1], 2, 6).value(cols[2])
    p.launch()
    api.scan_check()
    assert int(res.item()) == int((few[m] * bursts[m]).sum())


@pytest.mark.parametrize("n", [2_000, 70_000])
def test_short_sequences_corrupt(cuda, n):
    # flipped bytes either decode to other values or are reported, and the
    # library works afterwards
    r = np.random.default_rng(n)
    v, x = r.integers(0, 11, n), r.integers(0, 100, n)
    cx = _col(x, "none")
    reported = 0
    for trial in range(16):
        col = api.Column(v.astype(np.int32), "lz4", rows_per_chunk=40_000, lz4_min_match=4)
        pay = col.payload_view()
        b = col.blocks()[trial % col.info.n_blocks]
        at = int(b[0]) + int(r.integers(0, int(b[2])))
        pay[at] = 255 if trial % 2 else int(r.integers(0, 256))
        col.to_device()
        try:
            _sum(cuda, col, 2, 8, cx)
        except api.L.GxError as e:
            assert e.status == L.GX_ERR_CORRUPT
            reported += 1
    assert reported >= 1
    assert _sum(cuda, _col(v, "lz4", lz4_min_match=4), 2, 8, cx) == int(x[(v >= 2) & (v <= 8)].sum())
