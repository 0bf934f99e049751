"""Parquet page headers whose counts cannot be true are refused on the host: a
negative number of values, which another page of the chunk makes up for, would
place rows before and behind the output; level bytes of a version 2 page that
are negative or more than its uncompressed size would move its values out of
the page."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import GfpdbError, ops, parquet_writer
from flexpushdowndb_gb300.tupleset import Column, Table

TABLE = Table([Column("a", "int32", np.arange(1000))])


def written(monkeypatch, header):
    monkeypatch.setattr(parquet_writer, "_page_header", header)
    return np.frombuffer(parquet_writer.write_parquet(TABLE, page_rows=500, dictionary_max=0), dtype=np.uint8)


@pytest.mark.parametrize("counts", [(-5, 1005), (1000 - (1 << 31) + 500, (1 << 31) - 500), (-1, 1001)])
def test_negative_values(monkeypatch, counts):
    plain, left = parquet_writer._page_header, list(counts)
    data = written(monkeypatch, lambda kind, size, n, enc: plain(kind, size, left.pop(0), enc))
    with pytest.raises(GfpdbError, match="negative"):
        ops.parquet_layout(data)


def test_negative_dictionary(monkeypatch):
    plain = parquet_writer._page_header
    monkeypatch.setattr(parquet_writer, "_page_header",
                        lambda kind, size, n, enc: plain(kind, size, -n if kind == 2 else n, enc))
    data = np.frombuffer(parquet_writer.write_parquet(TABLE, page_rows=500), dtype=np.uint8)
    with pytest.raises(GfpdbError, match="negative"):
        ops.parquet_layout(data)


@pytest.mark.parametrize("levels,uncompressed,fragment", [(-8, 2000, "negative"), (2000, 1000, "levels"),
                                                          (0, 2000, None), (40, 2000, None)])
def test_version_2_levels(monkeypatch, levels, uncompressed, fragment):
    def header(kind, size, n, enc):
        w = parquet_writer._Compact()
        w.i32(1, 3)
        w.i32(2, uncompressed)
        w.i32(3, size)
        w.begin_struct(8)
        w.i32(1, n)
        w.i32(2, 0)
        w.i32(3, n)
        w.i32(4, enc)
        w.i32(5, levels)
        w.i32(6, 0)
        w.end_struct()
        w.out.append(0)
        return bytes(w.out)

    data = written(monkeypatch, header)
    if fragment is None:
        assert [p["numValues"] for p in ops.parquet_layout(data)["pages"]] == [500, 500]
    else:
        with pytest.raises(GfpdbError, match=fragment):
            ops.parquet_layout(data)
