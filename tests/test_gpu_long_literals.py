"""LZ4 columns of many short matches with stretches of literals among them: a
literal run belongs to one token wherever it ends, so a token met in a short
segment may announce hundreds of words.  Every scan form gives numpy's sums."""
import numpy as np
import pytest

from golap_public_b200 import _lib as L
from golap_public_b200 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _auto_form():
    yield
    api.set_scan_form("auto")


def _sequences(col):
    """(sequences of the column, longest literal run in words), read from its LZ4 blocks."""
    pay, count, longest = col.payload_view(), 0, 0
    for off, size in col.blocks()[:, [0, 2]].astype(np.int64):
        b = pay[off:off + size].tobytes()
        p = 0
        while p < len(b):
            tok = b[p]
            p += 1
            lit = tok >> 4
            if lit == 15:
                while b[p] == 255:
                    lit += 255
                    p += 1
                lit += b[p]
                p += 1
            p += lit
            count += 1
            longest = max(longest, lit // 4)
            if p >= len(b):
                break
            p += 2
            if tok & 15 == 15:
                while b[p] == 255:
                    p += 1
                p += 1
    return count, longest


def _column(r, n, seg, stretch, where):
    """Values of few distinct ones; every 4096 rows (8192 for the longest) a stretch that does not repeat, starting
    in some segment's first, middle or last row, or across the end of a tile and of the smallest blocks."""
    v = r.integers(0, 11 if seg > 32 else 7, n).astype(np.int64)
    wide = r.permutation(1 << 20)[:n] + 1000
    for k, base in enumerate(range(0, n, 4096 if stretch < 1000 else 8192)):
        at = base + seg * (3 + k) + {"first": 0, "middle": seg // 2 + 1, "last": seg - 1, "end": 0}[where]
        if where == "end":
            at = base + 4096 - stretch // 2
        v[at:at + stretch] = wide[at:at + stretch]
    return v


@pytest.mark.parametrize("where", ["first", "middle", "last", "end"])
@pytest.mark.parametrize("stretch", [70, 131, 132, 133, 200, 700, 2000])
@pytest.mark.parametrize("rpb,seg", [(4096, 32), (8192, 64), (16384, 128)])
def test_long_literals(cuda, rpb, seg, stretch, where):
    n = 70_003
    r = np.random.default_rng(seg * 10_000 + stretch)
    v, w, price = _column(r, n, seg, stretch, where), _column(r, n, seg, 5, "middle"), r.integers(0, 2**31, n)
    kw = dict(rows_per_chunk=40_000, rows_per_block=rpb, lz4_segments=rpb // seg)
    cv, cw = (api.Column(x.astype(np.int32), "lz4", lz4_min_match=4, **kw).to_device() for x in (v, w))
    cp = api.Column(price.astype(np.int32), "lz4", **kw).to_device()
    seqs, longest = _sequences(cv)
    assert longest >= stretch // 2  # (a block end may cut it)
    assert seqs * 8 >= n * 3  # many sequences: the single-plan scan decodes it with one lane per segment
    m = (v >= 1) & (v <= 2000)
    want = int(price[m].sum()), int((w[m] * v[m]).sum()), int(v[w >= 2].sum())
    res = cuda.zeros(3, dtype=cuda.int64, device="cuda")
    for form in ("warp", "pipe", "shared", "queue"):
        api.set_scan_form(form)
        res.zero_()
        api.ScanPlan(agg=L.GX_AGG_SUM, result=res[0:]).filter(cv, 1, 2000).value(cp).launch()
        api.ScanPlan(agg=L.GX_AGG_SUM_PRODUCT, result=res[1:]).filter(cv, 1, 2000, carry=True).value(cw).launch()
        api.ScanPlan(agg=L.GX_AGG_SUM, result=res[2:]).filter(cw, 2, 1 << 21).value(cv).launch()
        api.scan_check()
        assert tuple(res.tolist()) == want, form
