"""Segmented LZ4 columns on both sides of the rule that picks the group decoder
(many short sequences: a warp's groups in step): the decompressed column and
every scan form's sum against numpy, with long literal runs, long and
overlapping matches, one to 128 segments a block, ragged tiles."""
import numpy as np
import pytest

from golap_public_b200 import _lib as L
from golap_public_b200 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _auto_form():
    yield
    api.set_scan_form("auto")


def _values(kind, n):
    r = np.random.default_rng(n)
    runs = lambda k, hi: np.repeat(r.integers(0, hi, n // k + 1), k)[:n]
    at = np.arange(n)
    return {"small": lambda: r.integers(0, 11, n), "wide": lambda: r.integers(0, 60, n), "runs4": lambda: runs(4, 99),
            "runs5": lambda: runs(5, 99), "runs8": lambda: runs(8, 1000), "runs300": lambda: runs(300, 1000),
            "sparse": lambda: np.where(r.random(n) < .05, r.integers(0, 10**6, n), 0),
            "tile3": lambda: np.where((at // 64) % 2 == 0, at % 3, r.integers(0, 9, n)),
            "bursts": lambda: np.where((at // 400) % 3 == 0, r.integers(0, 10**6, n), 7),
            "half": lambda: np.where((at // 4000) % 2 == 0, r.integers(0, 9, n), runs(90, 99))}[kind]()


@pytest.mark.parametrize("kind", ["small", "wide", "runs4", "runs5", "runs8", "runs300", "sparse", "tile3", "bursts",
                                  "half"])
@pytest.mark.parametrize("rpb,S", [(16384, 128), (16384, 16), (16384, 8), (4096, 128)])
@pytest.mark.parametrize("n", [33, 70_003])
def test_density(cuda, kind, rpb, S, n):
    v = _values(kind, n)
    w = np.random.default_rng(1).integers(0, 1000, n)
    for match in (4, 12):
        col = api.Column(v.astype(np.int32), "lz4", rows_per_chunk=40_000, rows_per_block=rpb, lz4_segments=S,
                         lz4_min_match=match).to_device()
        other = api.Column(w.astype(np.int32), "none", rows_per_chunk=40_000, rows_per_block=rpb).to_device()
        out = cuda.empty(n, dtype=cuda.int32, device="cuda")
        api.ChunkDecompressor(col).chunks(0, col.info.n_chunks, out)
        api.scan_check()
        assert (out.cpu().numpy() == v).all()
        lo, hi = int(np.quantile(v, 0.2)), int(np.quantile(v, 0.8))
        want = int(w[(v >= lo) & (v <= hi)].sum()), int(v[w >= 500].sum())
        res = cuda.zeros(2, dtype=cuda.int64, device="cuda")
        for form in ("warp", "pipe", "shared", "queue"):
            if form in ("warp", "shared", "pipe") and rpb // S > 1024:
                continue  # (segments longer than a tile)
            api.set_scan_form(form)
            res.zero_()
            api.ScanPlan(agg=L.GX_AGG_SUM, result=res[0:]).filter(col, lo, hi).value(other).launch()
            api.ScanPlan(agg=L.GX_AGG_SUM, result=res[1:]).filter(other, 500, 999).value(col).launch()
            api.scan_check()
            assert tuple(res.tolist()) == want, (form, match)
