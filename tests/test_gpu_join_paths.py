"""Join-table builds and probes at the edges of their four-row batches: sizes
around a batch and a CTA, unaligned arrays, duplicate and reserved keys, rows
dropped by predicates, tables filled to the last slot."""
import numpy as np
import pytest

from golap_public_b200 import _lib as L
from golap_public_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["linear", "bucket", "dense"])
@pytest.mark.parametrize("n", [1, 3, 5, 1023, 1025, 70_001, 200_003])
@pytest.mark.parametrize("shift", [0, 1])
def test_build_and_probe(cuda, layout, n, shift):
    r = np.random.default_rng(n + shift)
    keys = r.permutation(n).astype(np.int32) - n // 3
    reg, reg2 = r.integers(0, 4, n).astype(np.int32), r.integers(0, 9, n).astype(np.int32)
    pay = r.integers(-2**31, 2**31, n).astype(np.int32)

    def dev(a):  # `shift` words off a 16-byte boundary
        t = cuda.zeros(len(a) + 4, dtype=cuda.int32, device="cuda")
        t[shift:shift + len(a)] = cuda.from_numpy(a).cuda()
        return t[shift:shift + len(a)]

    ht = api.HashMap(n, layout)
    kd, pd, rd, r2 = dev(keys), dev(pay), dev(reg), dev(reg2)
    probe = r.integers(-n, 2 * n, 3 * n + 1).astype(np.int32)
    qd = dev(probe)
    for payload, preds, ok in ((pd, [(rd, 1, 2)], (reg >= 1) & (reg <= 2)), (None, [], np.ones(n, bool)),
                               (pd, [(rd, 0, 2), (r2, 3, 8)], (reg <= 2) & (reg2 >= 3))):
        ht.build(kd, payload, preds=preds)
        assert ht.count() == int(ok.sum())
        val = pay if payload is not None else np.arange(n, dtype=np.int32)
        look = np.full(4 * n + 4, -2**31, np.int64)
        look[keys[ok] + n] = val[ok]
        want = look[probe + n]
        hit = np.isin(probe, keys[ok])
        out, hits = dev(np.zeros_like(probe)), cuda.zeros(1, dtype=cuda.int64, device="cuda")
        ht.probe(qd, out, hits)
        assert int(hits.item()) == int(hit.sum())
        assert (out.cpu().numpy() == np.where(hit, want, -2**31)).all()
        hits.zero_()
        ht.probe(qd, None, hits)
        assert int(hits.item()) == int(hit.sum())


@pytest.mark.parametrize("layout", ["linear", "bucket", "dense"])
def test_duplicates_reserved_and_full(cuda, layout):
    # every key three times, a reserved key among them: the first insert of each
    # wins somewhere among its rows; then as many keys as the table has slots
    k = np.repeat(np.arange(1000, dtype=np.int32), 3)
    ht = api.HashMap(1000, layout)
    ht.build(cuda.from_numpy(k).cuda(), None)
    assert ht.count() == 1000
    out = cuda.zeros(1000, dtype=cuda.int32, device="cuda")
    ht.probe(cuda.arange(1000, dtype=cuda.int32, device="cuda"), out)
    assert (out.cpu().numpy() // 3 == np.arange(1000)).all()
    k[7] = -2**31
    ht.build(cuda.from_numpy(k).cuda(), None)
    with pytest.raises(L.GxError) as e:
        ht.count()
    assert e.value.status == L.GX_ERR_CAPACITY
    full = np.arange(16, dtype=np.int32) * 7
    small = api.HashMap(8, layout)  # 16 slots in the hashed layouts
    small.build(cuda.from_numpy(full).cuda(), None)
    hits = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    small.probe(cuda.arange(-50, 200, dtype=cuda.int32, device="cuda"), None, hits)
    assert int(hits.item()) == 16
