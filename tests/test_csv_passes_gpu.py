"""The CSV passes where they can go wrong, against the oracle: fields that
start before their tile (just, far, and whole tiles before), tiles with more
separators than one part holds, string groups larger than a warp's staging
buffer, every alignment of a string's source and place, numbers of every
length around the eight digits converted at once, signs, quotes, carriage
returns, empty fields, and 1 to 256 fields a line."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import GfpdbError, ops
from oracle import ops as oops

pytestmark = pytest.mark.gpu

FIELDS = [("a", "int64"), ("s", "utf8"), ("p", "decimal(15,2)"), ("d", "date32"), ("u", "utf8"), ("b", "int32")]


def check(text, fields, **kw):
    got = ops.csv_read(text, fields, **kw)
    want = oops.csv_parse(text, fields, **kw)
    assert got.names == want.names
    assert got.rows() == want.rows()


def lines(rows, widths, seed, end="\n"):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(rows):
        s, u = ("x" * int(rng.choice(widths)) for _ in range(2))
        s = "".join(chr(97 + (i * 7 + len(s)) % 26) for i in range(len(s)))
        if rng.integers(0, 5) == 0:
            u = f'"{u}"'
        digits = int(rng.integers(1, 16))
        a = rng.choice(["", "-", "+"]) + str(rng.integers(10 ** (digits - 1), 10**digits))
        p = rng.choice(["", "-"]) + f"{rng.integers(0, 10 ** int(rng.integers(1, 12)))}.{rng.integers(0, 100):02d}"
        day = f"{rng.integers(1600, 2400)}-{rng.integers(1, 13):02d}-{rng.integers(1, 29):02d}"
        out.append("|".join([a, s, p, day, u, str(rng.integers(-(10**9), 10**9))]))
    return (end.join(out) + end).encode()


@pytest.mark.parametrize("rows,widths,end", [
    (700, [0, 1, 2, 3, 5, 17], "\n"), (700, [0, 33, 63, 64, 65, 66], "\r\n"), (300, [100, 255, 256, 257, 300], "\n"),
    (60, [5, 16_383, 16_384, 40_000], "\n"), (1, [3], "\n"), (4000, [10, 25, 40], "\n"),
])
def test_fields_and_strings(gpu, rows, widths, end):
    text = lines(rows, widths, rows + len(widths), end)
    check(text, FIELDS, delimiter="|")
    check(text[: -len(end)], FIELDS, delimiter="|", has_header=False)  # unterminated
    check(b"h|h|h|h|h|h\n" + text, FIELDS, delimiter="|", has_header=True, columns=["u", "p", "s"])


@pytest.mark.parametrize("fields", [1, 2, 3, 255, 256])
@pytest.mark.parametrize("ty", ["int32", "utf8"])
def test_dense_text(gpu, fields, ty):
    """One-digit and empty fields: tiles of 8,192 to 16,384 separators."""
    fs = [(f"f{i}", ty) for i in range(fields)]
    emit = [f"f{i}" for i in sorted({0, fields // 2, fields - 1})]
    rng = np.random.default_rng(fields)
    v = rng.integers(0, 10, 40_000 // fields * fields).reshape(-1, fields)
    text = "\n".join(",".join("" if ty == "utf8" and x == 0 else str(x) for x in row) for row in v).encode()
    check(text, fs, delimiter=",", columns=emit)
    check(text + b"\n", fs, delimiter=",", columns=emit)
    if ty == "utf8":
        check(b"," * (fields - 1) + (b"\n" + b"," * (fields - 1)) * (20_000 // fields) + b"\n", fs, delimiter=",",
              columns=emit)


@pytest.mark.parametrize("bad,ty", [("", "int32"), ("-", "int64"), ("12345x78", "int64"), ("1234567890123x", "int64"),
                                    ("99999999999", "int32"), ("1.234", "decimal(15,2)"), ("1.2.3", "decimal(15,2)"),
                                    (".", "decimal(15,2)"), ("1:.00", "decimal(15,2)"), ("123456789.0/", "decimal(15,2)"),
                                    ("1992-13-01", "date32"), ("1992-01-00", "date32"), ("1992/01/01", "date32"),
                                    ("19920-1-01", "date32"), ("1992-01-1", "date32")])
def test_malformed_fields(gpu, bad, ty):
    good = {"int32": "7", "int64": "7", "decimal(15,2)": "7.00", "date32": "1999-12-31"}[ty]
    rows = [f"{good}|k{i}" for i in range(3000)]
    check("\n".join(rows).encode(), [("v", ty), ("k", "utf8")], delimiter="|")
    rows[1777] = f"{bad}|k"
    with pytest.raises(GfpdbError, match="malformed CSV.*row 1777"):
        ops.csv_read("\n".join(rows).encode(), [("v", ty), ("k", "utf8")], delimiter="|")


@pytest.mark.parametrize("text,value", [(b".50", 50), (b"-.50", -50), (b"+3", 300), (b"3.", 300), (b"3.5", 350),
                                        (b"12345678.99", 1234567899), (b"123456789.99", 12345678999)])
def test_decimal_forms(gpu, text, value):
    assert ops.csv_read(text + b"\n", [("p", "decimal(15,2)")], delimiter="|")["p"].tolist() == [value]
