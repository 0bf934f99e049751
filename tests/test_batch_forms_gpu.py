"""Batched star queries at the edges of the direct fact pass's staged forms
and of the two ways the result is gathered, against the oracle: foreign keys
at and past the ends of a dimension's key range (the ends of int32 too),
dimensions small enough for a mask per key, too large for it and too large to
stage, 1 to 64 queries, and group tables on both sides of the one-launch
limit."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import batch, plan, workloads
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table
from oracle import queries

pytestmark = pytest.mark.gpu


def run(tabs, parts, qs, **kw):
    spec = workloads.star_batch_spec(parts, qs, **kw)
    inputs = plan.PreparedInputs({k: DeviceTable.from_host(v) for k, v in tabs.items()})
    want = {q: queries.star_query_ranges(tabs, parts, r).sorted_rows() for q, r in enumerate(qs)}
    for got in (batch.star_batch(spec, inputs), batch.PreparedBatch(spec, inputs).execute()):
        rows = batch.split_by_query(got.table)
        assert {q: rows.get(q, []) for q in want} == want
        ids = [r[0] for r in got.table.rows()]
        assert ids == sorted(ids)  # each query's rows together


def tables(dim_rows, first, sizes, seed):
    rng = np.random.default_rng(seed)
    tabs = {}
    for i, (n, k0) in enumerate(zip(dim_rows, first), 1):
        tabs[f"d{i}"] = Table([Column(f"d{i}_pk", "int32", k0 + rng.permutation(n)),
                               Column(f"d{i}_f", "int32", rng.integers(0, 100, n)),
                               Column(f"d{i}_g", "int32", rng.integers(0, 10, n))])
    for p, rows in enumerate(sizes):
        cols = []
        for i, (n, k0) in enumerate(zip(dim_rows, first), 1):
            fk = k0 + rng.integers(0, n, rows)
            odd = rng.random(rows) < 0.05  # just outside the range, and the ends of int32
            ends = np.array([k0 - 1, k0 + n, -(1 << 31), (1 << 31) - 1])
            fk[odd] = np.clip(ends[rng.integers(0, 4, odd.sum())], -(1 << 31), (1 << 31) - 1)
            cols.append(Column(f"fk{i}", "int32", fk))
        cols += [Column("qty", "int32", rng.integers(1, 50, rows)),
                 Column("price_cents", "int64", rng.integers(-(1 << 61), 1 << 61, rows)),
                 Column("discount", "int32", rng.integers(0, 11, rows))]
        tabs[f"p{p}"] = Table(cols)
    return tabs, [f"p{p}" for p in range(len(sizes))]


@pytest.mark.parametrize("dim_rows,first", [
    ((3, 17, 200, 1), (-(1 << 31), (1 << 31) - 17, -100, (1 << 31) - 1)),
    ((2000, 30_000, 64, 5000), (1, 1, 1, 1)), ((60_000, 70_000, 50_000, 40_000), (-30_000, 5, 0, -40_000)),
])
@pytest.mark.parametrize("n_queries", [1, 7, 32, 64])
def test_staged_forms(gpu, dim_rows, first, n_queries):
    tabs, parts = tables(dim_rows, first, [130_003, 0, 511, 1], n_queries)
    qs = workloads.batch_queries(n_queries, seed=n_queries)
    for blocks in (1, 4):
        run(tabs, parts, qs, blocks_per_sm=blocks, groups_hint=4096)


@pytest.mark.parametrize("hint", [100, 8192, 8193, 40_000])
def test_group_table_sizes(gpu, hint):
    tabs, parts = tables((500, 900, 700, 800), (1, 1, 1, 1), [20_000, 3000], 3)
    run(tabs, parts, workloads.batch_queries(5, seed=9), groups_hint=hint)
