"""A probe whose output array is its key array, one key per lane and four."""
import numpy as np
import pytest

from golap_public_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["linear", "bucket", "dense"])
@pytest.mark.parametrize("n", [7, 16_384, 16_385, 300_001, 3_000_000])
@pytest.mark.parametrize("shift", [0, 1])
def test_probe_in_place(cuda, layout, n, shift):
    r = np.random.default_rng(n)
    keys = r.permutation(20_000).astype(np.int32)
    pay = r.integers(-2**31, 2**31, 20_000).astype(np.int32)
    ht = api.HashMap(20_000, layout)
    kd, pd = cuda.from_numpy(keys).cuda(), cuda.from_numpy(pay).cuda()
    ht.build(kd, pd)
    probe = r.integers(0, 30_000, n).astype(np.int32)
    buf = cuda.empty(n + 4, dtype=cuda.int32, device="cuda")[shift:shift + n]
    look = np.full(30_000, -2**31, np.int32)
    look[keys] = pay
    for hits in (None, cuda.zeros(1, dtype=cuda.int64, device="cuda")):
        buf.copy_(cuda.from_numpy(probe))
        ht.probe(buf, buf, hits)
        assert (buf.cpu().numpy() == look[probe]).all()
    assert int(hits.item()) == int((probe < 20_000).sum())
