"""Large group-by batches whose aggregates are counts and integer sums, minima
and maxima of plain columns, against sorted numpy reductions: one to four of
them in every order of adding and comparing ones, 32- and 64-bit and date
columns, one narrow, one wide and two narrow keys, few and many groups, row
counts around the warps' steps, the values at the ends of their ranges, and
float or computed aggregates beside them (which take the general kernel)."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.expression import col, plus
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu

LARGE = 2 << 20


def table(rows, groups, seed):
    rng = np.random.default_rng(seed)
    key = rng.integers(0, groups, rows)
    v = rng.integers(-(1 << 63), 1 << 63, rows, dtype=np.int64)
    v[rng.integers(0, rows, 50)] = np.iinfo(np.int64).min
    v[rng.integers(0, rows, 50)] = np.iinfo(np.int64).max
    q = rng.integers(-(1 << 31), 1 << 31, rows).astype(np.int32)
    q[:2] = np.iinfo(np.int32).min, np.iinfo(np.int32).max
    return Table([Column("k", "int32", key - groups // 2), Column("w", "int64", (key - 3) * 0x1E3779B97F4A7C15),
                  Column("a", "int32", key // 1000 - 5), Column("b", "int32", key % 1000),
                  Column("v", "int64", v), Column("q", "int32", q), Column("d", "date32", rng.integers(0, 9000, rows)),
                  Column("f", "float64", rng.integers(0, 9, rows).astype(np.float64)), Column("id", "int64", key)])


def check(t, keys, aggs):
    specs = [ops.aggregate(fn, f"x{i}", None if c is None else plus(col("v"), col("q")) if c == "vq" else col(c))
             for i, (fn, c) in enumerate(aggs)]
    g = ops.Group(keys, specs)
    g.group(DeviceTable.from_host(Table([x for x in t.columns if x.name != "id"])))
    got = g.finalise()
    order = np.argsort(t["id"], kind="stable")
    key = t["id"][order]
    first = np.flatnonzero(np.r_[True, key[1:] != key[:-1]])
    names = keys + [f"x{i}" for i in range(len(aggs))]
    cols = [t[k][order][first].astype(np.int64) for k in keys]
    with np.errstate(over="ignore"):
        for fn, c in aggs:
            x = np.ones(t.num_rows, np.int64) if c is None else t["v"] + t["q"] if c == "vq" else t[c]
            x = x if x.dtype == np.float64 else x.astype(np.int64)
            cols.append({"SUM": np.add, "COUNT": np.add, "MIN": np.minimum, "MAX": np.maximum}[fn].reduceat(x[order], first))
    at = np.lexsort([np.asarray(got[k], np.int64) for k in reversed(keys)])
    want_at = np.lexsort([c for c in reversed(cols[: len(keys)])])
    for name, want in zip(names, cols):
        assert np.array_equal(np.asarray(got[name])[at].astype(want.dtype), want[want_at]), name


KINDS = [[("MIN", "v")], [("SUM", "q")], [("COUNT", None), ("SUM", "v")], [("MAX", "v"), ("SUM", "v")],
         [("MIN", "q"), ("MAX", "d")], [("SUM", "v"), ("COUNT", None), ("SUM", "q")],
         [("MAX", "q"), ("MIN", "v"), ("COUNT", None)], [("MIN", "v"), ("MAX", "v"), ("MIN", "d")],
         [("SUM", "v"), ("SUM", "q"), ("SUM", "d"), ("COUNT", None)],
         [("MAX", "v"), ("SUM", "v"), ("MIN", "q"), ("COUNT", None)],
         [("SUM", "v"), ("MIN", "v"), ("SUM", "q"), ("COUNT", None)],
         [("SUM", "f"), ("COUNT", None)], [("SUM", "vq"), ("MAX", "q")]]


@pytest.mark.parametrize("aggs", KINDS, ids=lambda a: "-".join(f"{f}{c}" for f, c in a))
@pytest.mark.parametrize("groups", [40, 900_000])
def test_kinds(gpu, aggs, groups):
    check(table(LARGE + 37, groups, groups), ["w"], aggs)


@pytest.mark.parametrize("keys", [["k"], ["w"], ["a", "b"]])
@pytest.mark.parametrize("rows", [LARGE, LARGE + 1, LARGE + 31, LARGE + 32, LARGE + 33, LARGE + 63, LARGE + 2047, 5_000_001])
def test_keys_and_rows(gpu, keys, rows):
    check(table(rows, 200_000, rows % 97), keys, [("SUM", "v"), ("COUNT", None), ("MAX", "q")])


@pytest.mark.parametrize("aggs", [[("SUM", "v"), ("COUNT", None), ("MAX", "q")], [("MIN", "v"), ("SUM", "q")]],
                         ids=["3", "2"])
@pytest.mark.parametrize("groups", [1, 7, 5000, 150_000])
@pytest.mark.parametrize("rows", [(3 << 16) - 1, 3 << 16, (3 << 16) + 1, 152 * 2048 - 1, 152 * 2048, 152 * 2048 + 1])
def test_smallest_batches(gpu, rows, groups, aggs):
    """Batches around the size from which they take the plain kernel, and
    around one step of every block."""
    check(table(rows, groups, rows % 89), ["w"], aggs)
