"""Join probes of tables on both sides of the size that is kept in the L1
(16,384 slots), with runs that go past a key's first group (high load factors,
repeated build keys), for batches around a warp's 32 rows and the 512 matches
that a warp stages."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key", ["int32", "int64"])
@pytest.mark.parametrize("build,times,load,rows", [
    (8192, 1, 0.5, 70_001), (8193, 1, 0.5, 70_001), (14_745, 1, 0.9, 70_001), (14_746, 1, 0.9, 70_001),
    (1, 1, 0.5, 1), (1, 1, 0.5, 31), (1, 1, 0.5, 33), (3, 1, 0.9, 20_000), (1, 40, 0.5, 513), (900, 9, 0.9, 30_000),
    (5000, 7, 0.9, 30_000),
])
def test_probe(gpu, key, build, times, load, rows):
    rng = np.random.default_rng(build + rows)
    stride = 1 if key == "int32" else (1 << 33) + 1
    bk = np.repeat(rng.permutation(build), times)
    b = Table([Column("bk", key, bk * stride), Column("bv", "int32", np.arange(bk.size))])
    pk = rng.integers(0, max(2, build + build // 2), rows)
    p = Table([Column("pk", key, pk * stride), Column("pv", "int32", np.arange(rows))])
    j = ops.HashJoin("bk", "pk", ["pv", "bv"], load_factor=load)
    j.put_build(DeviceTable.from_host(b))
    j.finalize_build()
    got = j.probe(DeviceTable.from_host(p))
    order = np.argsort(bk, kind="stable")
    first = np.searchsorted(bk[order], pk)
    hit = pk < build
    want = np.stack([np.repeat(np.flatnonzero(hit), times),
                     order[(first[hit][:, None] + np.arange(times)).reshape(-1)]], axis=1)
    have = np.stack([got["pv"], got["bv"]], axis=1)
    assert np.array_equal(have[np.lexsort(have.T)], want[np.lexsort(want.T)])
