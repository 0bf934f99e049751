"""The prefix sum behind string gathers and ordered joins, at sizes around its
tiles (2,048 and 8,192 values), the size where they change and the look-back's
windows of 128 tiles: a join that keeps every probe row places each row by it."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 128 * 2048, 128 * 2048 + 1, 257 * 2048 + 5, (1 << 19) - 1, 1 << 19,
                               (1 << 19) + 1, 128 * 8192 - 3, 129 * 8192 + 7, 3_000_001])
def test_probe_rows_in_order(gpu, n):
    rng = np.random.default_rng(n)
    build = Table([Column("bk", "int64", np.repeat(np.arange(40), np.arange(40) % 4)),
                   Column("bv", "int32", np.arange(sum(i % 4 for i in range(40))))])
    key = rng.integers(0, 50, n)
    probe = Table([Column("pk", "int64", key), Column("pv", "int32", np.arange(n))])
    j = ops.HashJoin("bk", "pk", ["pv", "bv"], join_type="RIGHT_SEMI")
    j.put_build(DeviceTable.from_host(build))
    j.finalize_build()
    got = j.probe(DeviceTable.from_host(probe))["pv"]
    assert np.array_equal(np.sort(got), np.flatnonzero((key < 40) & (key % 4 > 0)))
    j = ops.HashJoin("bk", "pk", ["pv"], join_type="LEFT")
    j.put_build(DeviceTable.from_host(build))
    j.finalize_build()
    got = j.probe(DeviceTable.from_host(probe))["pv"]
    times = np.where(key < 40, key % 4, 0)
    assert np.array_equal(np.sort(got), np.repeat(np.arange(n), times))
