"""Dictionary-encoded Parquet pages of several parts whose indices come in many
runs: runs of one length (found many at a step), of lengths that all differ
(more of them than a batch's walk takes, so that their parts are decoded in the
read's second round), RLE runs between bit-packed ones, in one and in several
batches of chunks, with a damaged run before and after where a walk stops,
against the values written. Bit for bit."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import GfpdbError, ops, parquet_writer
from flexpushdowndb_gb300.parquet_writer import write_parquet
from flexpushdowndb_gb300.tupleset import Column, Table

pytestmark = pytest.mark.gpu


def _pack(idx, bw):
    padded = np.zeros((len(idx) + 7) // 8 * 8, dtype=np.uint32)
    padded[: len(idx)] = idx
    bits = ((padded[:, None] >> np.arange(bw, dtype=np.uint32)) & 1).astype(np.uint8).reshape(-1)
    return np.packbits(bits, bitorder="little").tobytes()


def _runs(lengths):
    """A page's indices as bit-packed runs of the lengths (multiples of 8), in
    turn; 0: an RLE run of as many as repeat, where at least two do."""

    def write(idx, bw):
        out, at, k = bytearray([bw]), 0, 0
        while at < len(idx):
            n = lengths[k % len(lengths)]
            k += 1
            w = parquet_writer._Compact()
            if n == 0:
                same = 1
                while at + same < len(idx) and idx[at + same] == idx[at] and same < 900:
                    same += 1
                if same < 2:
                    continue
                w.varint(same << 1)
                out += bytes(w.out) + int(idx[at]).to_bytes((bw + 7) // 8, "little")
                at += same
                continue
            w.varint((min(n, (len(idx) - at + 7) // 8 * 8) // 8 << 1) | 1)
            out += bytes(w.out) + _pack(idx[at : at + n], bw)
            at += n
        return bytes(out)

    return write


def _table(rows, distinct, plain):
    rng = np.random.default_rng(rows)
    code = rng.integers(0, distinct, rows)
    cols = [Column("i", "int32", code * 7 - 3), Column("l", "int64", code * (1 << 33) + 1),
            Column("u", "utf8", np.array([f"v{c}" for c in range(distinct)])[code].tolist())]
    if plain:  # fills batches of chunks
        cols.append(Column("p", "int64", rng.integers(0, 1 << 62, rows)))
    return Table(cols)


def _same(got, t):
    assert got.names == t.names
    for g, w in zip(got.columns, t.columns):
        if w.type == "utf8":
            assert g.to_list() == w.to_list()
        else:
            assert np.array_equal(g.values, w.values), g.name


VARIED = [8 * (1 + (i * 37) % 29) for i in range(61)]


@pytest.mark.parametrize("lengths,rows,group,page,distinct,plain", [
    (n, *size, False) for n in ([8], [504], [1024], [16, 0], VARIED, VARIED + [0])
    for size in ((8193, 8193, 8193, 7), (300_000, 300_000, 300_000, 40), (70_000, 70_000, 9000, 3000))
] + [(n, 3_000_000, 1_000_000, 500_000, 250, True) for n in ([504], VARIED)])
def test_many_runs(gpu, monkeypatch, lengths, rows, group, page, distinct, plain):
    monkeypatch.setattr(parquet_writer, "_bitpacked", _runs(lengths))
    t = _table(rows, distinct, plain)
    data = np.frombuffer(write_parquet(t, row_group_rows=group, page_rows=page), dtype=np.uint8)
    assert not plain or len(data) > 3 * (8 << 20)
    _same(ops.parquet_read(data), t)
    _same(ops.parquet_read(data, ["u", "i"]), Table([t.column("u"), t.column("i")]))


@pytest.mark.parametrize("lengths", [[504], VARIED])
@pytest.mark.parametrize("share", [0.01, 0.5, 0.999])
def test_damaged_run(gpu, monkeypatch, lengths, share):
    """A run header that claims more values than the page has bytes for."""
    monkeypatch.setattr(parquet_writer, "_bitpacked", _runs(lengths))
    t = _table(600_000, 200, False)
    data = np.frombuffer(write_parquet(t, row_group_rows=600_000, page_rows=600_000), dtype=np.uint8)
    page = [p for p in ops.parquet_layout(data, ["i"])["pages"] if p["pageType"] == 0][-1]
    heads, k = [1], 0  # where the run headers lie behind the page's header
    while heads[-1] < page["compressedBytes"]:
        n = lengths[k % len(lengths)] // 8
        heads.append(heads[-1] + (1 if n < 64 else 2) + n * 8)
        k += 1
    at = page["offset"] + heads[int(share * (len(heads) - 2))]
    bad = data.copy()
    bad[at : at + 4] = [0xFF, 0xFF, 0xFF, 0x7F]
    with pytest.raises(GfpdbError, match="malformed Parquet page data"):
        ops.parquet_read(bad, ["i"])
    _same(ops.parquet_read(data), t)
