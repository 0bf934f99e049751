"""Dictionary-encoded Parquet pages whose indices several CTAs decode (8,192
values each): page sizes around the parts' edges, one long bit-packed run or
many RLE and bit-packed runs that start and end inside, on and across those
edges, index widths of 1 to 17 bits, every column type, against the values
written. Bit for bit."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops, parquet_writer
from flexpushdowndb_gb300.parquet_writer import write_parquet
from flexpushdowndb_gb300.tupleset import Column, Table

pytestmark = pytest.mark.gpu

PACK = parquet_writer._bitpacked


def _mixed_runs(idx, bw):
    """The indices as runs of uneven length: a stretch of one value as an RLE
    run, the others bit-packed (multiples of 8 values but the last)."""
    out, at, k = bytes([bw]), 0, 0
    rng = np.random.default_rng(len(idx))
    while at < len(idx):
        same = 1
        while at + same < len(idx) and idx[at + same] == idx[at]:
            same += 1
        if same >= 16 or at + same == len(idx):
            w = parquet_writer._Compact()
            w.varint(same << 1)
            out += bytes(w.out) + int(idx[at]).to_bytes((bw + 7) // 8, "little")
            at += same
        else:
            n = 8 * int(rng.integers(1, 120))
            out += PACK(idx[at : at + n], bw)[1:]
            at += n
        k += 1
    return out


def _table(rows, distinct, seed):
    rng = np.random.default_rng(seed)
    code = rng.integers(0, distinct, rows)
    code[: min(rows, distinct)] = np.arange(min(rows, distinct))  # every value occurs
    for lo in range(0, rows, 5000):  # stretches of one value, some across a part's edge
        code[lo + 3000 : lo + 3300] = code[lo]
    return Table([Column("i", "int32", code * 7 - 3), Column("l", "int64", code * (1 << 33) + 1),
                  Column("f", "float64", code * 0.37), Column("t", "date32", code),
                  Column("u", "utf8", [f"v{c}" for c in code])])


@pytest.mark.parametrize("runs", ["one", "mixed"])
@pytest.mark.parametrize("rows,page_rows,distinct", [(8191, 8191, 2), (8192, 8192, 3), (8193, 8193, 200),
                                                      (40_000, 24_577, 5_000), (70_001, 70_001, 69_000), (5, 5, 1)])
def test_parts_of_a_page(gpu, monkeypatch, runs, rows, page_rows, distinct):
    if runs == "mixed":
        monkeypatch.setattr(parquet_writer, "_bitpacked", _mixed_runs)
    t = _table(rows, distinct, rows + distinct)
    data = write_parquet(t, row_group_rows=1 << 20, page_rows=page_rows, dictionary_max=1 << 17)
    got = ops.parquet_read(np.frombuffer(data, dtype=np.uint8))
    assert got.names == t.names
    for g, w in zip(got.columns, t.columns):
        if w.type == "utf8":
            assert g.to_list() == w.to_list()
        else:
            assert np.array_equal(g.values.view(np.uint8), w.values.view(np.uint8)), g.name
