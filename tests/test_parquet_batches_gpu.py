"""Parquet reads of several batches of column chunks (more than 8 MB each), the
next one copied while one is decoded, against the values written: pageable and
page-locked files, columns in another order than the file's, row ranges by
file position, and a damaged page in the last batch."""

import numpy as np
import pytest
import torch

from flexpushdowndb_gb300 import GfpdbError, ops
from flexpushdowndb_gb300.parquet_writer import write_parquet
from flexpushdowndb_gb300.tupleset import Column, Table

pytestmark = pytest.mark.gpu

ROWS = 900_000


@pytest.fixture(scope="module")
def made():
    rng = np.random.default_rng(8)
    code = rng.integers(0, 3000, ROWS)
    words = np.array([f"word{i}" * (1 + i % 3) for i in range(3000)])
    t = Table([Column("i", "int32", rng.integers(0, 1 << 30, ROWS)), Column("l", "int64", rng.integers(0, 1 << 60, ROWS)),
               Column("u", "utf8", words[code].tolist()), Column("k", "int32", code),
               Column("f", "float64", rng.normal(0, 1, ROWS)), Column("m", "int64", np.arange(ROWS))])
    return t, np.frombuffer(write_parquet(t, row_group_rows=200_000, page_rows=70_000), dtype=np.uint8)


def same(got, t, names, lo=0, hi=ROWS):
    assert got.names == names
    want = t.slice(lo, hi)
    for n in names:
        a, b = got[n], want[n]
        assert np.array_equal(np.asarray(a), np.asarray(b)), n


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("names", [None, ["m", "u", "i"], ["l"], ["f", "k", "l", "m", "u"]])
def test_batches(gpu, made, pinned, names):
    t, data = made
    assert len(data) > 3 * (8 << 20)
    if pinned:
        held = torch.from_numpy(data.copy()).pin_memory()
        data = held.numpy()
    same(ops.parquet_read(data, names), t, names or t.names)


def test_row_groups_by_position(gpu, made):
    t, data = made
    at = [g["offset"] for g in ops.parquet_layout(data)["rowGroups"]]
    same(ops.parquet_read(data, None, at[1], at[3]), t, t.names, 200_000, 800_000)


def test_damage_in_the_last_batch(gpu, made):
    t, data = made
    pages = ops.parquet_layout(data, ["k"])["pages"]
    last = [p for p in pages if p["pageType"] == 0][-1]
    bad = data.copy()
    bad[last["offset"]] = 200  # an index width of 200 bits
    with pytest.raises(GfpdbError, match="malformed Parquet page data"):
        ops.parquet_read(bad)
    same(ops.parquet_read(data, ["k"]), t, ["k"])  # the next read is not affected
