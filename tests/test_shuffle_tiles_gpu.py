"""Shuffles at the edges of tiles (2,048 and 4,096 rows), of warps (256 rows)
and of the slot counts that change a launch, against a stable sort by slot:
one integer key of each width, a composite key with strings, every column
width, more columns than one launch takes, and all rows in one slot."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.tupleset import Column, Table
from oracle import ops as oops

pytestmark = pytest.mark.gpu

BIG = 152 * 2 * 16 * 256  # from here on 152 SMs get two tiles of 4,096 rows each


def check(t, keys, slots):
    got, offs = ops.shuffle(t, keys, slots)
    slot = oops.shuffle_slots(t, keys, slots)
    order = np.argsort(slot, kind="stable")
    assert offs == np.concatenate([[0], np.cumsum(np.bincount(slot, minlength=slots))]).tolist()
    for name in t.names:
        assert np.array_equal(np.asarray(got[name]), np.asarray(t[name])[order]), name


@pytest.mark.parametrize("ty", ["int32", "int64"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 2047, 2048, 2049, 3 * 2048 + 1025])
@pytest.mark.parametrize("slots", [1, 2, 31, 32, 33, 255, 256, 257, 1023, 1024])
def test_tiles(gpu, n, slots, ty):
    rng = np.random.default_rng(n + slots)
    check(Table([Column("k", ty, rng.integers(-3000, 3000, n)), Column("f", "float64", rng.normal(0, 1, n)),
                 Column("row", "int32", np.arange(n))]), ["k"], slots)


@pytest.mark.parametrize("n", [BIG - 1, BIG, BIG + 4097])
@pytest.mark.parametrize("slots", [2, 256, 1024])
def test_large_tiles(gpu, n, slots):
    rng = np.random.default_rng(slots)
    check(Table([Column("k", "int32", rng.integers(0, 1 << 30, n)), Column("row", "int64", np.arange(n))]), ["k"], slots)


@pytest.mark.parametrize("n", [5000, BIG + 1])
def test_one_slot_takes_all(gpu, n):
    check(Table([Column("k", "int64", np.full(n, 7)), Column("row", "int32", np.arange(n))]), ["k"], 300)


def test_columns_past_one_launch(gpu):
    """Strings through the inverse permutation, 30 columns of both widths, a
    composite key."""
    n = 9001
    rng = np.random.default_rng(2)
    cols = [Column("s", "utf8", [f"w{i}" for i in rng.integers(0, 99, n)])]
    cols += [Column(f"c{i}", "int64" if i % 2 else "int32", rng.integers(0, 1 << 20, n)) for i in range(30)]
    check(Table(cols), ["s", "c3"], 77)
