"""Group-key digits out of range are an error for rows that are alive at their
step, and only for those -- also where the column, or another step's, holds one
value on a tile and is decided for all of its rows at once."""
import numpy as np
import pytest

from golap_public_b200 import _lib as L
from golap_public_b200 import api

pytestmark = pytest.mark.gpu
T = 1024  # rows of a tile
N = 8 * T
FORMS = ["warp", "pipe", "shared", "queue"]


@pytest.fixture(autouse=True)
def _auto_form():
    yield
    api.set_scan_form("auto")


def _table(torch, keys, payload, layout="linear"):
    dev = [torch.from_numpy(np.asarray(x, np.int32)).cuda() for x in (keys, payload)]
    return api.HashMap(len(keys), layout).build(*dev), dev


def _plan(torch, kind, codec, year, drop):
    """A plan of the given kind over N rows: `year` (cascaded) is one value on every tile, with digits 1993..1994;
    `drop` rows are dropped by a step before it.  Returns the plan, its group table and what to keep alive."""
    col = lambda v, c: api.Column(v.astype(np.int32), c, rows_per_chunk=5 * T, rows_per_block=T).to_device()
    r = np.random.default_rng(1)
    v = r.integers(1, 1000, N)
    cy, cv = col(year, "cascaded"), col(v, "none")
    key = np.where(drop, 9, r.integers(1, 4, N))  # key 9 is in no table
    ck = col(key, codec)
    date, keep_date = _table(torch, [1992, 1993, 1994], [1992, 1993, 1994])
    dim, keep_dim = _table(torch, [1, 2, 3], [0, 1, 2], "dense")
    agg = api.HashAggregate(64)
    p = api.ScanPlan(agg=L.GX_AGG_SUM, groupby=agg)
    group = (year - 1993).astype(np.int64)
    if kind == "group":
        p.filter(ck, 1, 3).group(cy, 1993, 2).value(cv)
    elif kind == "run-time":
        p.filter(ck, 1, 3).filter(ck, 0, 5).group(cy, 1993, 2).value(cv)
    elif kind == "q2":
        p.probe(ck, dim, 0, 3).probe(ck, dim).probe(cy, date, 1993, 2).value(cv)
        group += 2 * (key - 1)
    elif kind == "q3":
        p.probe(ck, dim, 0, 3).probe(ck, dim, 0, 3).probe(cy, date, 1993, 2).value(cv)
        group += 2 * (key - 1) + 6 * (key - 1)
    else:  # q4, minus a carried column of zeros
        p.agg = L.GX_AGG_SUM_DIFF
        cz = col(np.zeros(N, np.int64), "none")
        p.probe(ck, dim, 0, 3).probe(ck, dim).probe(cy, date, 1993, 2).probe(ck, dim).carry(cz).value(cv)
        group += 2 * (key - 1)
    ok = ~drop & (year >= 1993)
    want = {int(g): int(v[ok & (group == g)].sum()) for g in np.unique(group[ok])}
    return p, agg, want, (keep_date, keep_dim)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("codec", ["none", "lz4", "cascaded"])
@pytest.mark.parametrize("kind", ["group", "run-time", "q2", "q3", "q4"])
def test_digit_of_a_constant_column(cuda, kind, codec, form):
    if form == "queue" and kind == "q4":
        pytest.skip("the queue form takes no plan with a carried column and digits")
    api.set_scan_form(form)
    year = np.repeat([1992, 1993, 1994, 1992, 1993, 1994, 1993, 1992], T)
    drop = (year == 1992) | (np.arange(N) % 3 == 0)  # no row with a digit out of range is alive at the step
    p, agg, want, keep = _plan(cuda, kind, codec, year, drop)
    p.launch()
    api.scan_check()
    assert agg.read() == want
    for at in (3 * T, 4 * T - 1):  # one row is
        drop[at] = False
        p, agg, _, keep = _plan(cuda, kind, codec, year, drop)
        p.launch()
        with pytest.raises(L.GxError) as e:
            api.scan_check()
        assert e.value.status == L.GX_ERR_INVALID
        drop[at] = True


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("digit", ["rows", "constant"])
def test_digit_before_a_constant_step_that_drops_the_tile(cuda, digit, form):
    # the digit's step comes first: its rows are alive there, whatever a later step does to the tile
    api.set_scan_form(form)
    col = lambda v, c: api.Column(v.astype(np.int32), c, rows_per_chunk=5 * T, rows_per_block=T).to_device()
    day = np.repeat(np.arange(8), T)
    cd, cv = col(day, "cascaded"), col(np.ones(N), "none")
    for last, bad in ((5, False), (6, True)):
        k = np.where(day == 3, last, 2) if digit == "constant" else np.full(N, 2)
        if digit == "rows":
            k[np.arange(N) % 2 == 0] = 4
            k[3 * T + 77] = last
        agg = api.HashAggregate(64)
        p = api.ScanPlan(agg=L.GX_AGG_SUM, groupby=agg)
        p.group(col(k, "cascaded" if digit == "constant" else "none"), 0, 6).filter(cd, 4, 7).value(cv)
        p.launch()
        if bad:
            with pytest.raises(L.GxError) as e:
                api.scan_check()
            assert e.value.status == L.GX_ERR_INVALID
        else:
            api.scan_check()
            m = day >= 4
            assert agg.read() == {int(g): int((k[m] == g).sum()) for g in np.unique(k[m])}
