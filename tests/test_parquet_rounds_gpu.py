"""Parquet reads of several batches whose pages are not decoded with their batch:
compressed pages, inflated together, and byte arrays whose lengths are walked in
the read's second round, as dictionaries and as plain pages, against the values
written. Bit for bit."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import GfpdbError, ops, parquet_writer
from flexpushdowndb_gb300.parquet_writer import write_parquet
from flexpushdowndb_gb300.tupleset import Column, Table

pytestmark = pytest.mark.gpu

ROWS = 1_600_000


def snappy(monkeypatch):
    """The writer's pages as snappy blocks of literals and its column chunks'
    codec with them."""
    plain, bits, header, compact = (getattr(parquet_writer, n) for n in ("_plain", "_bitpacked", "_page_header", "_Compact"))
    sizes = {}

    def block(body):
        w = compact()
        w.varint(len(body))
        out = bytearray(w.out)
        for at in range(0, len(body), 60_000):
            part = body[at : at + 60_000]
            out += bytes([61 << 2]) + (len(part) - 1).to_bytes(2, "little") + part
        sizes[len(out)] = len(body)
        return bytes(out)

    class Coded(compact):
        def i32(self, fid, v):
            super().i32(fid, 1 if (fid, v) == (4, 0) else v)  # a column chunk's codec

    def start(kind, uncompressed, size):
        w = compact()
        w.i32(1, kind)
        w.i32(2, uncompressed)
        w.i32(3, size)
        return bytes(w.out)

    def coded_header(kind, size, n, enc):
        return start(kind, sizes[size], size) + header(kind, size, n, enc)[len(start(kind, size, size)) :]

    monkeypatch.setattr(parquet_writer, "_plain", lambda ty, v: block(plain(ty, v)))
    monkeypatch.setattr(parquet_writer, "_bitpacked", lambda idx, bw: block(bits(idx, bw)))
    monkeypatch.setattr(parquet_writer, "_page_header", coded_header)
    monkeypatch.setattr(parquet_writer, "_Compact", Coded)


@pytest.fixture(scope="module")
def table():
    rng = np.random.default_rng(4)
    code = rng.integers(0, 700, ROWS)
    words = np.array([f"w{i}" * (1 + i % 3) for i in range(700)])
    return Table([Column("l", "int64", rng.integers(0, 1 << 60, ROWS)), Column("u", "utf8", words[code].tolist()),
                  Column("k", "int32", code), Column("v", "utf8", words[(code * 7) % 90].tolist())])


def same(got, t):
    assert got.names == t.names
    for g, w in zip(got.columns, t.columns):
        assert g.to_list() == w.to_list() if w.type == "utf8" else np.array_equal(g.values, w.values), g.name


@pytest.mark.parametrize("compressed", [False, True])
@pytest.mark.parametrize("dictionary_max", [1 << 15, 0])
def test_rounds(gpu, monkeypatch, table, compressed, dictionary_max):
    if compressed:
        snappy(monkeypatch)
    data = np.frombuffer(write_parquet(table, row_group_rows=200_000, page_rows=10_000, dictionary_max=dictionary_max),
                         dtype=np.uint8)
    assert len(data) > 2 * (8 << 20)
    layout = ops.parquet_layout(data)
    assert {p["codec"] for p in layout["pages"]} == {1 if compressed else 0}
    same(ops.parquet_read(data), table)
    same(ops.parquet_read(data, ["v", "l"]), Table([table.column("v"), table.column("l")]))
    # a damaged length in the last page whose lengths are walked
    page = [p for p in layout["pages"] if layout["columns"][p["column"]]["name"] == "u" and p["numValues"] > 1
            and (p["pageType"] == 2 or dictionary_max == 0)][-1]
    bad = data.copy()
    at = page["offset"] + (8 if compressed else 0)  # behind a block's length and first tag
    bad[at : at + 4] = [0xFF, 0xFF, 0xFF, 0x7F]
    with pytest.raises(GfpdbError, match="malformed Parquet page data"):
        ops.parquet_read(bad)
    same(ops.parquet_read(data, ["u"]), Table([table.column("u")]))
