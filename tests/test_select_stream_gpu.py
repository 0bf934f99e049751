"""Selections over inputs of more than a million rows (two passes), against
numpy: every comparison on 32- and 64-bit columns, literals outside int32 on
an int32 column, ORs within clauses, rows around a warp's slice and a range of
slices, columns on 16- but not 32-byte boundaries, few, many and no rows
selected, and more output columns than one."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.expression import and_, col, eq, gt, gte, lt, lte, neq, num_lit, or_
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu

N = (1 << 20) + 65536 * 2 + 257


@pytest.fixture(scope="module")
def table():
    rng = np.random.default_rng(5)
    return Table([Column("a", "int32", rng.integers(0, 1000, N)), Column("b", "int64", rng.integers(-(1 << 40), 1 << 40, N)),
                  Column("d", "date32", rng.integers(8000, 9000, N)), Column("f", "float64", rng.normal(0, 1, N)),
                  Column("row", "int32", np.arange(N))])


def device(t, skip):
    """t's rows from `skip` on, in memory that starts `skip` rows later."""
    dt = DeviceTable.from_host(t)
    return DeviceTable(dt.names, dt.types, [[x[skip:] for x in ts] for ts in dt.tensors], t.num_rows - skip)


def check(t, pred, want, skip=0, rows=None):
    rows = t.num_rows - skip if rows is None else rows
    t = t.slice(0, skip + rows)
    got = ops.select(device(t, skip), ops.Filter(pred, t), project=["f", "row", "b"])
    at = np.nonzero(want[: skip + rows])[0]
    at = at[at >= skip]
    assert np.array_equal(got["row"], t["row"][at])
    assert np.array_equal(got["f"], t["f"][at]) and np.array_equal(got["b"], t["b"][at])


OPS = {"lt": (lt, np.less), "lte": (lte, np.less_equal), "gt": (gt, np.greater), "gte": (gte, np.greater_equal),
       "eq": (eq, np.equal), "neq": (neq, np.not_equal)}


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("name,ty,lit", [("a", "int32", 500), ("a", "int32", 0), ("a", "int64", 1 << 40),
                                         ("a", "int64", -(1 << 40)), ("b", "int64", 12345), ("d", "int32", 8999)])
def test_one_leaf(gpu, table, op, name, ty, lit):
    e, f = OPS[op]
    check(table, e(col(name), num_lit(lit, ty)), f(table[name], lit))


@pytest.mark.parametrize("skip", [0, 4, 8, 12])
@pytest.mark.parametrize("rows", [1 << 20, (1 << 20) + 1, (1 << 20) + 7, (1 << 20) + 249, (1 << 20) + 256, N - 12])
def test_clauses(gpu, table, skip, rows):
    a, b, d = table["a"], table["b"], table["d"]
    pred = and_(or_(lt(col("a"), num_lit(100)), gte(col("b"), num_lit(1 << 39, "int64")), eq(col("d"), num_lit(8500))),
                gt(col("d"), num_lit(8100)), or_(neq(col("a"), num_lit(7)), lt(col("b"), num_lit(0, "int64"))))
    want = ((a < 100) | (b >= 1 << 39) | (d == 8500)) & (d > 8100) & ((a != 7) | (b < 0))
    check(table, pred, want, skip, rows)


@pytest.mark.parametrize("lim", [-1, 0, 1, 998, 999])
def test_few_to_all(gpu, table, lim):
    check(table, and_(lte(col("a"), num_lit(lim)), gte(col("b"), num_lit(-(1 << 41), "int64"))), table["a"] <= lim)
