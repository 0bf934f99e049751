"""The places that the prefix sum gives to the rows of outer joins: a RIGHT join
keeps every probe row, each row's matches (or its one row without) beside its
neighbours' in the probe's order, at sizes around the sum's tiles (2,048 and
8,192 values) and the look-back's windows."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 128 * 2048, 128 * 2048 + 1, 257 * 2048 + 5, (1 << 19) - 1, 1 << 19,
                               (1 << 19) + 1, 128 * 8192 - 3, 129 * 8192 + 7, 2_000_001])
def test_kept_probe_rows_in_order(gpu, n):
    rng = np.random.default_rng(n)
    times = np.arange(40) % 4  # matches of each key; 0 and keys from 40 on: none
    build = Table([Column("bk", "int64", np.repeat(np.arange(40), times)), Column("bv", "int32", np.arange(times.sum()) + 1)])
    key = rng.integers(0, 50, n)
    probe = Table([Column("pk", "int64", key), Column("pv", "int32", np.arange(n))])
    first = np.cumsum(times) - times
    m = np.where(key < 40, times[np.minimum(key, 39)], 0)
    for join_type in ("RIGHT", "LEFT"):
        j = ops.HashJoin("bk", "pk", ["pv", "bv"], join_type=join_type)
        j.put_build(DeviceTable.from_host(build))
        j.finalize_build()
        got = j.probe(DeviceTable.from_host(probe))
        rows = np.maximum(m, 1) if join_type == "RIGHT" else m
        pv, bv = np.asarray(got["pv"]), np.array([0 if v is None else v for v in got.column("bv").to_list()])
        assert np.array_equal(pv, np.repeat(np.arange(n), rows))
        # a probe row's own matches in any order
        order = np.lexsort((bv, pv))
        k = np.arange(rows.sum()) - np.repeat(np.cumsum(rows) - rows, rows)
        want = np.where(np.repeat(m, rows) > 0, np.repeat(first[np.minimum(key, 39)], rows) + k + 1, 0)
        assert np.array_equal(bv[order], want)
