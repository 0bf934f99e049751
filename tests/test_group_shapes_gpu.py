"""Group-by at the edges of its block shapes and table layouts, against sorted
numpy reductions: batches just below and at the size that runs one large CTA
per SM, few, many and all-different keys, one hot key, sums that wrap and
carry between their halves, the all-ones key, no aggregate to eight, and
tables whose slots lie packed (one and three accumulators, a million slots and
more), grown from separate ones over several batches."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.expression import col, plus
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu

LARGE = 2 << 20

AGGS = [("SUM", "v"), ("COUNT", None), ("MAX", "q"), ("MIN", "v"), ("MAX", "v"), ("MIN", "q"), ("SUM", "q"), ("SUM", "vq")]


def spec(n):
    out = []
    for i, (fn, c) in enumerate(AGGS[:n]):
        e = None if c is None else plus(col("v"), col("q")) if c == "vq" else col(c)
        out.append(ops.aggregate(fn, f"a{i}", e))
    return out


def expected(key, v, q, n):
    order = np.argsort(key, kind="stable")
    key, v, q = key[order], v[order], q[order]
    first = np.flatnonzero(np.r_[True, key[1:] != key[:-1]])
    out = [key[first]]
    with np.errstate(over="ignore"):
        for fn, c in AGGS[:n]:
            x = np.ones_like(v) if c is None else v + q if c == "vq" else v if c == "v" else q.astype(np.int64)
            op = {"SUM": np.add, "COUNT": np.add, "MIN": np.minimum, "MAX": np.maximum}[fn]
            out.append(op.reduceat(x, first))
    return out


def data(rows, keys, seed):
    rng = np.random.default_rng(seed)
    if keys == "hot":  # one key on half the rows, the others seen once or twice
        k = np.where(rng.integers(0, 2, rows) == 0, 7, rng.integers(0, rows, rows))
    elif keys == "all":
        k = rng.permutation(rows)
    else:
        k = rng.integers(0, keys, rows)
    k = k * 0x1E3779B97F4A7C15  # scattered, wrapping
    k[rng.integers(0, rows, 5)] = -1  # the all-ones key
    v = rng.integers(-(1 << 62), 1 << 62, rows) | rng.integers(0, 2, rows) * 0xFFFFFFFF
    return k.astype(np.int64), v.astype(np.int64), rng.integers(-(1 << 31), 1 << 31, rows).astype(np.int32)


def run(batches, n):
    g = ops.Group(["k"], spec(n))
    for k, v, q in batches:
        g.group(DeviceTable.from_host(Table([Column("k", "int64", k), Column("v", "int64", v), Column("q", "int32", q)])))
    t = g.finalise()
    got = [c.values for c in t.columns]
    order = np.argsort(got[0], kind="stable")
    want = expected(*(np.concatenate(x) for x in zip(*batches)), n)
    for g_, w in zip(got, want):
        assert np.array_equal(g_[order].astype(np.int64), w)


@pytest.mark.parametrize("rows", [1, 31, 33, 256, 257, 4097, LARGE - 1, LARGE, LARGE + 31])
@pytest.mark.parametrize("keys", [3, 5000, "hot"])
def test_rows_and_keys(gpu, rows, keys):
    run([data(rows, keys, rows % 1000)], 3)


@pytest.mark.parametrize("n", [0, 1, 2, 4, 5, 8])
@pytest.mark.parametrize("rows", [70_000, LARGE])
def test_aggregate_counts(gpu, rows, n):
    run([data(rows, 9000, n)], n)


@pytest.mark.parametrize("n", [1, 2, 3])
def test_packed_tables_and_growth(gpu, n):
    run([data(LARGE, "all", 1)], n)
    run([data(1000, 400, 2), data(300_000, "all", 3), data(LARGE + 5, 3_000_000, 4)], n)


def test_narrow_key_pairs(gpu):
    rng = np.random.default_rng(5)
    a, b = rng.integers(-3, 3, LARGE).astype(np.int32), rng.integers(-40, 40, LARGE).astype(np.int32)
    t = Table([Column("a", "int32", a), Column("b", "int32", b), Column("v", "int64", np.arange(LARGE))])
    g = ops.Group(["a", "b"], [ops.aggregate("SUM", "s", col("v")), ops.aggregate("COUNT", "n")])
    g.group(DeviceTable.from_host(t))
    got = {(x, y): (s, c) for x, y, s, c in g.finalise().rows()}
    code = (a.astype(np.int64) + 3) * 80 + b + 40
    n, s = np.bincount(code, minlength=480), np.bincount(code, weights=np.arange(LARGE), minlength=480)
    assert got == {(i // 80 - 3, i % 80 - 40): (int(s[i]), int(n[i])) for i in range(480) if n[i]}
