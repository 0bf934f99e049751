"""CSV texts of one to nine string columns (up to four, several warps share a
column of a tile), with strings around what a warp's buffer holds for 32 rows
(48 bytes on average), long ones, empty ones, and fields that start before
their tile, against the oracle."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from oracle import ops as oops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("rows,widths", [(9000, [0, 1, 2, 3]), (3000, [40, 47, 48, 49, 56]), (1500, [0, 1, 60, 100, 131]),
                                         (200, [0, 300, 999, 1537]), (40, [3, 5000, 33_000]), (5, [1, 70_000]), (1, [40])])
def test_string_columns(gpu, columns, rows, widths):
    rng = np.random.default_rng(columns * 100 + rows)
    fields = [("k", "int32")] + [(f"s{i}", "utf8") for i in range(columns)]
    n = max(1, rows // columns)
    alphabet = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz0123456789", dtype=np.uint8)
    lines = []
    for r in range(n):
        strings = [alphabet[rng.integers(0, 36, int(w))].tobytes() for w in rng.choice(widths, columns)]
        lines.append(b"|".join([str(r).encode()] + strings))
    for text in (b"\n".join(lines), b"h|" * columns + b"h\n" + b"\n".join(lines) + b"\n"):
        header = text.startswith(b"h|")
        got = ops.csv_read(text, fields, delimiter="|", has_header=header)
        want = oops.csv_parse(text, fields, delimiter="|", has_header=header)
        assert got.names == want.names
        assert got.rows() == want.rows()
