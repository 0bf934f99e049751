"""Float64, computed and no aggregates in batches the general update kernel
takes: warps whose rows all go to one group (their float sums are added up in
registers), groups on both sides of what the shared-memory table holds, rows
sent straight to the global table (a large groupsHint), and the sizes around
which warps, blocks and the table's sizing change. The values are small whole
numbers, so every sum is exact in whatever order it is made."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.expression import col, times
from flexpushdowndb_gb300.ops import aggregate
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu

AGGS = {
    "none": [],
    "one": [("SUM", "f")],
    "two": [("SUM", "f"), ("SUM", "vq")],
    "six": [("SUM", "f"), ("MIN", "f"), ("MAX", "f"), ("COUNT", None), ("SUM", "vq"), ("SUM", "f2")],
}
EXPR = {"f": col("f"), "f2": times(col("f"), col("f")), "vq": times(col("v"), col("q"))}


def expected(fn, x, key, n):
    out = np.zeros(n, dtype=np.int64 if x is None or x.dtype == np.int64 else np.float64)
    if fn == "COUNT":
        return np.bincount(key, minlength=n)
    if fn == "SUM":
        np.add.at(out, key, x)
        return out
    out[:] = np.inf if fn == "MIN" else -np.inf
    (np.minimum if fn == "MIN" else np.maximum).at(out, key, x)
    return out


@pytest.mark.parametrize("aggs", list(AGGS))
@pytest.mark.parametrize("rows,keys,hint", [(1, 1, 0), (31, 1, 0), (33, 2, 0), (4097, 1, 0), (5000, 3, 5000), (70_001, 500, 0),
                                            (70_001, 30_000, 0), (70_001, 30_000, 40_000), ((2 << 20) - 1, 1, 0),
                                            ((2 << 20) + 33, 40, 0), ((2 << 20) + 33, 5000, 0)])
def test_general_update(gpu, aggs, rows, keys, hint):
    rng = np.random.default_rng(rows + keys)
    key = rng.integers(0, keys, rows)
    key[: min(rows, 96)] = keys - 1  # whole warps of one group in every case
    f, v, q = rng.integers(-50, 51, rows).astype(np.float64), rng.integers(-1000, 1001, rows), rng.integers(1, 51, rows)
    x = {"f": f, "f2": f * f, "vq": v * q, None: None}
    t = Table([Column("k", "int64", key * 1_000_003 - 5), Column("f", "float64", f), Column("v", "int64", v),
               Column("q", "int32", q)])
    g = ops.Group(["k"], [aggregate(fn, f"a{i}", EXPR.get(c)) for i, (fn, c) in enumerate(AGGS[aggs])], groups_hint=hint)
    g.group(DeviceTable.from_host(t))
    got = g.finalise()
    at = (got["k"] + 5) // 1_000_003
    present = np.unique(key)
    assert np.array_equal(np.sort(at), present)
    for i, (fn, c) in enumerate(AGGS[aggs]):
        assert np.array_equal(got[f"a{i}"], expected(fn, x[c], key, keys)[at])


@pytest.mark.parametrize("rows", [1, 32, 64, 1000, (2 << 20) + 1])
def test_float_sum_without_keys(gpu, rows):
    f = np.random.default_rng(rows).integers(-50, 51, rows).astype(np.float64)
    for special, want in ((None, f.sum()), (np.inf, np.inf), (np.nan, np.nan)):
        x = f.copy()
        if special is not None:
            x[rows // 2] = special
        g = ops.Group([], [aggregate("SUM", "s", col("f")), aggregate("COUNT", "n")])
        g.group(DeviceTable.from_host(Table([Column("f", "float64", x)])))
        got = g.finalise()
        assert np.array_equal(got["s"], [want], equal_nan=True) and got["n"][0] == rows
