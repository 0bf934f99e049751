"""Batches over page-locked host tables read a foreign key over the link once a
row, also that of a dimension whose column the rows are grouped by and that is
too large to stage: the bytes the library counts, and the results against the
same batch over device tables."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import batch, plan, workloads
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu

ROWS = 200_000
DIMS = (500, 400, 120_000, 130_000)  # the last two are looked up in device memory


def tables(seed=1):
    rng = np.random.default_rng(seed)
    tabs = {}
    for i, n in enumerate(DIMS, 1):
        tabs[f"d{i}"] = Table([Column(f"d{i}_pk", "int32", rng.permutation(n) - 7), Column(f"d{i}_f", "int32", rng.integers(0, 100, n)),
                               Column(f"d{i}_g", "int32", rng.integers(0, 9, n))])
    cols = [Column(f"fk{i}", "int32", rng.integers(-7, n - 7, ROWS)) for i, n in enumerate(DIMS, 1)]
    tabs["p0"] = Table(cols + [Column("qty", "int32", rng.integers(1, 50, ROWS)),
                               Column("price_cents", "int64", rng.integers(1, 10**7, ROWS)),
                               Column("discount", "int32", rng.integers(0, 11, ROWS))])
    return tabs


def run(tabs, groups, queries, pinned):
    spec = workloads.star_batch_spec(["p0"], queries)
    spec["groupBy"] = [{"dimension": d, "column": f"d{d + 1}_g"} for d in groups]
    inputs = plan.PreparedInputs(tabs if pinned else {k: DeviceTable.from_host(v) for k, v in tabs.items()}, pinned=pinned)
    return batch.PreparedBatch(spec, inputs).execute()


@pytest.mark.parametrize("groups", [[2], [3], [2, 3], [3, 1], [0, 2], [0, 1], [3, 3]])
def test_groups_of_unstaged_dimensions(gpu, groups):
    tabs = tables()
    queries = [[(0, 99)] * 4, [(0, 60), (0, 99), (10, 70), (0, 50)]]
    want = run(tabs, groups, queries, False).table
    got = run(tabs, groups, queries, True)
    assert sorted(got.table.rows()) == sorted(want.rows())
    # every row reaches the groups: no more is read than for staged groups but the dimensions' own columns
    staged = run(tabs, [0, 1][: len(groups)], queries, True)
    assert abs(got.stats["h2d_bytes"] - staged.stats["h2d_bytes"]) <= 4 * 2 * max(DIMS)
