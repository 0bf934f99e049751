"""The work a program has gfpdb do, as cases that can be timed and compared.

Whole queries go through the Python API (batch.PreparedBatch,
plan.PreparedPlan, plan.execute); single operators through the C ABI of
include/gfpdb.h, as an engine embeds them: device-resident Arrow columns in,
device-resident Arrow columns out, taken up as torch tensors without a copy.
Joins and group-bys return their rows in no particular order, so a pass ends
as a program's own use of them does: joined rows go to their row's place,
groups to their key's, and the few groups of a star query fill a cube.
"""

from __future__ import annotations

import ctypes
import json
import math

import numpy as np
import torch

from flexpushdowndb_gb300 import _abi, batch, ops, plan, workloads
from flexpushdowndb_gb300.expression import and_, col, gte, lt, num_lit, to_json
from flexpushdowndb_gb300.ops import aggregate
from flexpushdowndb_gb300.tupleset import DeviceTable, new_output, utf8_encode

DEV = "cuda"
TORCH = {"int32": torch.int32, "int64": torch.int64, "date32": torch.int32, "float64": torch.float64}
CUBE_STAR = (25, 7)  # distinct d2_g x d4_g of the star queries
KEY_SCATTER = 0x1E3779B97F4A7C15  # odd: scatters numbers over 64 bits (wrapping), one to one
KEY_INVERSE = (pow(KEY_SCATTER, -1, 1 << 64) + (1 << 63)) % (1 << 64) - (1 << 63)
STAR_AGGS = ("revenue", "discount_revenue", "cnt")


def listed():
    return [
        # A dashboard's refresh: 32 variants of one star query over a
        # partitioned fact table in one batch (SSB-SF10-sized; the benchmark's
        # headline workload), at the settings its tuner picks.
        {"name": "batch_32q_60m", "kind": "batch", "parts": 64, "largest_part": 4_000_000, "queries": 32,
         "blocks_per_sm": 2},
        # What a request server runs as one batch: a few queries over a
        # quarter of the partitions, at the default settings.
        {"name": "batch_8q_15m", "kind": "batch", "parts": 16, "largest_part": 4_000_000, "queries": 8,
         "blocks_per_sm": 4},
        # One prepared star query with bloom predicate transfer, as a
        # statement that runs again and again (SSB-SF1-sized).
        {"name": "star_plan_6m", "kind": "star", "rows": 6_000_000},
        # An ad-hoc two-table join and group-by over a string column, its plan
        # seen once: every operator launched on its own.
        {"name": "two_table_1m", "kind": "two_table", "rows": 1_000_000, "dim_rows": 20_000},
        # A selective scan of a large table (a range conjunction, about 2%).
        {"name": "filter_40m", "kind": "filter", "rows": 40_000_000, "percent": 2.0},
        # A fact table joined to a dimension, both past the L2.
        {"name": "join_2m_x_20m", "kind": "join", "build": 2_000_000, "probe": 20_000_000, "key": "int32",
         "type": "INNER"},
        # An outer join: every build row kept, 64-bit keys.
        {"name": "join_left_300k_x_1m", "kind": "join", "build": 300_001, "probe": 1_000_003, "key": "int64",
         "type": "LEFT"},
        # The smallest call: a lookup join of a few thousand rows.
        {"name": "join_1k_x_10k", "kind": "join", "build": 1_000, "probe": 10_000, "key": "int64", "type": "INNER"},
        # A high-cardinality group-by with Zipf(1.1) keys.
        {"name": "group_20m", "kind": "group", "rows": 20_000_000, "keys": 10_000_000},
        # Loading text: lineitem-shaped lines, every field of them.
        {"name": "csv_2m", "kind": "csv", "rows": 2_000_000},
        # Loading a Parquet file that is in host memory.
        {"name": "parquet_4m", "kind": "parquet", "rows": 4_000_000, "page_rows": 131_072},
        # Spreading rows over the slots of a parallel plan.
        {"name": "shuffle_20m", "kind": "shuffle", "rows": 20_000_000, "slots": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["batch", "star", "two_table", "filter", "bloom", "join", "join", "group", "csv", "parquet",
                       "shuffle"])
    c = {"kind": kind}
    if kind == "batch":
        c |= {"parts": _log(rng, 1, 64), "largest_part": _log(rng, 100_000, 4_000_000), "queries": rng.randint(1, 32),
              "blocks_per_sm": rng.choice([2, 4])}
    elif kind == "star":
        c |= {"rows": _log(rng, 60_000, 6_000_000)}
    elif kind == "two_table":
        c |= {"rows": _log(rng, 10_000, 1_000_000), "dim_rows": _log(rng, 200, 20_000)}
    elif kind == "filter":
        c |= {"rows": _log(rng, 1_000, 40_000_000), "percent": round(math.exp(rng.uniform(0.0, math.log(50.0))), 1)}
    elif kind == "bloom":  # predicate transfer by hand: a filter over a dimension's keys, tested by a fact table
        c |= {"keys": _log(rng, 10, 50_000), "rows": _log(rng, 1_000, 1_000_000)}
    elif kind == "join":
        c |= {"build": _log(rng, 10, 2_000_000), "probe": _log(rng, 1_000, 20_000_000),
              "key": rng.choice(["int32", "int64"]), "type": rng.choice(["INNER", "INNER", "LEFT", "RIGHT_SEMI"])}
        if c["type"] != "INNER":
            c["probe"] = min(c["probe"], 2_000_000)
    elif kind == "group":
        c |= {"rows": _log(rng, 10_000, 20_000_000)}
        c["keys"] = _log(rng, 5, c["rows"] // 2)
    elif kind == "csv":
        c |= {"rows": _log(rng, 1_000, 2_000_000)}
    elif kind == "parquet":
        c |= {"rows": _log(rng, 10_000, 4_000_000), "page_rows": _log(rng, 5_000, 131_072)}
    else:
        c |= {"rows": _log(rng, 10_000, 20_000_000), "slots": _log(rng, 2, 1_024)}
    return c


# ------------------------------------------------------------------- inputs


class _Draw:
    """Random columns on the GPU, from the seed alone."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed) * 1_000_003 + 17)

    def ints(self, lo, hi, n, ty="int32"):
        """Uniform on [lo, hi]."""
        return torch.randint(int(lo), int(hi) + 1, (int(n),), generator=self.g, device=DEV, dtype=TORCH[ty])

    def order(self, n):
        return torch.randperm(int(n), generator=self.g, device=DEV)

    def unit(self, n):
        return torch.rand((int(n),), generator=self.g, device=DEV, dtype=torch.float64)


def _table(cols):
    """A DeviceTable of (name, type, tensor) columns."""
    return DeviceTable([c[0] for c in cols], [c[1] for c in cols], [[c[2]] for c in cols], cols[0][2].numel())


def _arange(n, start=0):
    return torch.arange(start, start + int(n), device=DEV, dtype=torch.int32)


def _star_dims(d, filter_values):
    out = {}
    for i, n in enumerate(workloads.STAR_DIM_ROWS):
        out[f"d{i + 1}"] = _table([
            (f"d{i + 1}_pk", "int32", _arange(n, 1)),
            (f"d{i + 1}_f", "int32", d.ints(0, filter_values[i] - 1, n)),
            (f"d{i + 1}_g", "int32", d.ints(0, workloads.STAR_GROUP_VALUES[i] - 1, n)),
        ])
    return out


def _star_fact(d, rows):
    cols = [(f"fk{i}", "int32", d.ints(1, n, rows)) for i, n in enumerate(workloads.STAR_DIM_ROWS, 1)]
    return _table(cols + [("qty", "int32", d.ints(1, 50, rows)),
                          ("price_cents", "int64", d.ints(90_000, 10_500_000, rows, "int64")),
                          ("discount", "int32", d.ints(0, 10, rows))])


def _part_sizes(c):
    return workloads.batch_partition_sizes(c["parts"], lo=min(50_000, c["largest_part"] // 2), hi=c["largest_part"])


def _digits(x):
    n = torch.ones_like(x)
    for k in range(1, 10):
        n += x >= 10**k
    return n


def _put_number(buf, pos, x, width):
    """Decimal digits of x right-aligned in the `width` bytes at pos."""
    for k in range(int(width.max())):
        m = width > k
        buf[(pos + width - 1 - k)[m]] = (48 + (x // 10**k) % 10)[m].to(torch.uint8)


def _lineitem_text(d, rows):
    """'|'-delimited text of workloads.LINEITEM_FIELDS, made on the GPU."""
    alphabet = torch.tensor(list(b"ABCDEFGHIJKLMNOPQRSTUVWXYZabcdefghijklmnopqrstuvwxyz0123456789 "), device=DEV,
                            dtype=torch.uint8)
    days = torch.arange(workloads.DATE_LO, workloads.DATE_HI + 1)
    ymd = torch.stack([torch.from_numpy(np.asarray(v)) for v in workloads.civil_from_days(days.numpy())]).to(DEV)
    fields, lens = [], []
    for _, ty in workloads.LINEITEM_FIELDS:
        if ty == "int32":
            v = d.ints(1, 1 << 20, rows, "int64")
            lens.append(_digits(v))
        elif ty.startswith("decimal"):
            v = d.ints(0, 10_000_000, rows, "int64")
            lens.append(_digits(v // 100) + 3)
        elif ty == "date32":
            v = d.ints(0, len(days) - 1, rows, "int64")
            lens.append(torch.full_like(v, 10))
        else:
            v = 10 + d.order(rows) % 31  # 10 to 40, as many bytes in all for every seed
            lens.append(v)
        fields.append((ty, v))
    row_len = sum(lens) + len(fields)
    off = torch.cumsum(row_len, 0) - row_len
    buf = torch.empty(int(row_len.sum()), device=DEV, dtype=torch.uint8)
    for f, (ty, v) in enumerate(fields):
        n = lens[f]
        if ty == "int32":
            _put_number(buf, off, v, n)
        elif ty.startswith("decimal"):
            _put_number(buf, off, v // 100, n - 3)
            buf[off + n - 3] = ord(".")
            _put_number(buf, off + n - 2, v % 100, torch.full_like(n, 2))
        elif ty == "date32":
            for k, (at, w) in enumerate(((0, 4), (5, 2), (8, 2))):
                _put_number(buf, off + at, ymd[k][v], torch.full_like(n, w))
            buf[off + 4] = ord("-")
            buf[off + 7] = ord("-")
        else:
            total = int(n.sum())
            first = torch.repeat_interleave(off - (torch.cumsum(n, 0) - n), n)
            buf[first + torch.arange(total, device=DEV)] = alphabet[d.ints(0, len(alphabet) - 1, total, "int64")]
        buf[off + n] = ord("|") if f + 1 < len(fields) else ord("\n")
        off = off + n + 1
    return buf


# --------------------------------------------- the C ABI with device results

_VIEW = {b"i": ("<i4", 4), b"l": ("<i8", 8), b"tdD": ("<i4", 4), b"g": ("<f8", 8)}


class _Owner:
    """An exported TupleSet, released with the last tensor over it."""

    def __init__(self, schema, array):
        self.schema, self.array = schema, array

    def __del__(self):
        if self.array.array.release:
            self.array.array.release(ctypes.pointer(self.array.array))
        if self.schema.release:
            self.schema.release(ctypes.pointer(self.schema))


class _View:
    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr or 0, False), "version": 3}


def _tensor(owner, ptr, n, typestr):
    if n == 0:
        return torch.empty(0, dtype={"<i4": torch.int32, "<i8": torch.int64, "<f8": torch.float64,
                                     "|u1": torch.uint8}[typestr], device=DEV)
    return torch.as_tensor(_View(owner, ptr, n, typestr), device=DEV)


def _taken(schema, array):
    """The columns of a device result as {name: tensor} (utf8: its offsets and
    bytes), in place."""
    owner = _Owner(schema, array)
    n = array.array.length
    out = {}
    for i in range(schema.n_children):
        cs, ca = schema.children[i].contents, array.array.children[i].contents
        name = cs.name.decode()
        if cs.format == b"u":
            offs = _tensor(owner, ca.buffers[1], n + 1, "<i4")
            out[name] = offs
            out[name + ".bytes"] = _tensor(owner, ca.buffers[2], int(offs[-1]), "|u1")
        else:
            out[name] = _tensor(owner, ca.buffers[1], n, _VIEW[cs.format][0])
    return out


def _call(fn, *args):
    _abi.check(fn(*args))


def _out(fn, *args):
    """fn(*args, out schema, out array, default stream) and its result."""
    s, a = new_output()
    _call(fn, *args, ctypes.byref(s), ctypes.byref(a), None)
    return _taken(s, a)


class _Handle:
    def __init__(self, free):
        self.h, self.free = ctypes.c_void_p(), free

    def __del__(self):
        if self.h.value:
            self.free(self.h)


# ---------------------------------------------------------------- the cases


def prepare(case, seed):
    c, d = case, _Draw(seed)
    st = {"case": c}
    kind = c["kind"]
    if kind == "batch":
        tabs = _star_dims(d, [workloads.BATCH_FILTER_VALUES] * 4)
        parts = [f"p{i}" for i in range(c["parts"])]
        for p, n in zip(parts, _part_sizes(c)):
            tabs[p] = _star_fact(d, n)
        st["tables"] = tabs
        st["queries"] = workloads.batch_queries(c["queries"], seed=int(seed) % 1_000_000)
        st["run"] = batch.PreparedBatch(workloads.star_batch_spec(parts, st["queries"],
                                                                  blocks_per_sm=c["blocks_per_sm"]), tabs)
    elif kind == "star":
        st["tables"] = _star_dims(d, workloads.STAR_FILTER_VALUES) | {"fact": _star_fact(d, c["rows"])}
        text = workloads.star_plan().to_json()
        st["run"] = plan.PreparedPlan(text[:-1] + ',"cudaGraph":true}', st["tables"])
        for _ in range(2):  # the runs that measure the plan and capture it
            st["run"].execute()
    elif kind == "two_table":
        offs, data = utf8_encode(workloads.REGIONS)
        width = len(workloads.REGIONS[0])
        region = d.ints(0, len(workloads.REGIONS) - 1, c["dim_rows"], "int64")
        chars = torch.from_numpy(data).to(DEV).reshape(-1, width)[region].reshape(-1)
        dim = DeviceTable(["pk", "category", "region"], ["int32", "int32", "utf8"],
                          [[_arange(c["dim_rows"], 1)],
                           [d.ints(0, 24, c["dim_rows"])],
                           [_arange(c["dim_rows"] + 1) * width, chars]],
                          c["dim_rows"])
        fact = _table([("fk", "int32", d.ints(1, c["dim_rows"], c["rows"])), ("qty", "int32", d.ints(1, 50, c["rows"])),
                       ("price_cents", "int64", d.ints(90_000, 10_500_000, c["rows"], "int64"))])
        st["tables"], st["region"] = {"fact": fact, "dim": dim}, region
        st["inputs"] = plan.PreparedInputs(st["tables"])
        st["text"] = workloads.two_table_plan().to_json()
    elif kind == "filter":
        n = c["rows"]
        # every input selects the same number of rows, at random places: the
        # others fail one half of the conjunction or the other, or both
        share = math.sqrt(c["percent"] / 100.0)
        a_lim, b_lim = round(1000 * share), round(10**9 * (1 - share))
        u = d.unit(n)
        fail = torch.where(u < 0.5 * (1 - share), 3, torch.where(u < 0.5, 1, 2))
        fail[d.order(n)[: round(n * c["percent"] / 100.0)]] = 0
        a = torch.where(fail & 1 == 0, d.ints(0, a_lim - 1, n), d.ints(a_lim, 999, n))
        b = torch.where(fail & 2 == 0, d.ints(b_lim, 10**9 - 1, n, "int64"), d.ints(0, b_lim - 1, n, "int64"))
        t = _table([("a", "int32", a), ("b", "int64", b), ("c", "int32", d.ints(0, 10**6, n)),
                    ("d", "int64", d.ints(-(10**12), 10**12, n, "int64"))])
        st["ex"] = t.export()
        st["filter"] = _Handle(_abi.lib().gfpdb_filter_free)
        pred = and_(lt(col("a"), num_lit(a_lim, "int32")), gte(col("b"), num_lit(b_lim, "int64")))
        _call(_abi.lib().gfpdb_filter_compile, to_json(pred).encode(), st["ex"].schema_ptr,
              ctypes.byref(st["filter"].h))
        st["names"] = _abi.cstr_array(["c", "d"])
    elif kind == "bloom":
        k, n = c["keys"], c["rows"]
        dim = _table([("b_0", "int64", d.ints(0, 2 * k, k, "int64")), ("b_1", "int64", d.ints(0, 1 << 40, k, "int64"))])
        fact = _table([("c_0", "int64", d.ints(0, 8 * k, n, "int64")), ("c_row", "int32", _arange(n)),
                       ("c_1", "int64", d.ints(0, 1 << 40, n, "int64")), ("c_2", "int32", d.ints(0, 1 << 20, n))])
        st["dim"], st["fact"] = dim.export(), fact.export()
        st["batches"] = (ctypes.POINTER(_abi.ArrowDeviceArray) * 1)(st["dim"].array_ptr)
        st["dim_key"], st["fact_key"] = _abi.cstr_array(["b_0"]), _abi.cstr_array(["c_0"])
    elif kind == "join":
        ty, nb, n = c["key"], c["build"], c["probe"]
        # unique build keys over twice their number, so about half the probe
        # rows find one
        stride = 1 if ty == "int32" else 1_000_003
        keys = (d.order(2 * nb)[:nb] * stride).to(TORCH[ty])
        b = _table([("b_row", "int32", _arange(nb)), ("b_key", ty, keys),
                    ("b_1", "int64", d.ints(0, 1 << 40, nb, "int64")), ("b_2", "int32", d.ints(0, 1 << 20, nb))])
        p = _table([("c_key", ty, (d.ints(0, 2 * nb - 1, n, "int64") * stride).to(TORCH[ty])),
                    ("c_row", "int32", _arange(n)),
                    ("c_1", "int64", d.ints(0, 1 << 40, n, "int64"))])
        st["b"], st["p"] = b.export(), p.export()
        st["bk"], st["pk"] = _abi.cstr_array(["b_key"]), _abi.cstr_array(["c_key"])
        st["needed"] = ["c_row", "c_1"]
        st["needed"] += {"INNER": ["b_1", "b_2"], "LEFT": ["b_row", "b_1"], "RIGHT_SEMI": []}[c["type"]]
        st["c_needed"] = _abi.cstr_array(st["needed"])
    elif kind == "group":
        n, k = c["rows"], c["keys"]
        cdf = np.cumsum(np.arange(1, k + 1, dtype=np.float64) ** -1.1)
        rank = torch.searchsorted(torch.from_numpy(cdf / cdf[-1]).to(DEV), d.unit(n)).clamp_(max=k - 1)
        key = (rank + 1) * KEY_SCATTER
        st["t"] = _table([("k", "int64", key), ("v", "int64", d.ints(-1_000_000, 1_000_000, n, "int64")),
                          ("q", "int32", d.ints(1, 50, n))])
        st["ex"] = st["t"].export()
        st["spec"] = _GROUP_SPEC
    elif kind == "csv":
        st["text"] = _lineitem_text(d, c["rows"])
        st["schema"], st["keep"] = _csv_schema(workloads.LINEITEM_FIELDS)
    elif kind == "parquet":
        from flexpushdowndb_gb300.parquet_writer import write_parquet

        data = write_parquet(workloads.star_fact(c["rows"], seed=int(seed) % 1_000_000), row_group_rows=1 << 20,
                             page_rows=c["page_rows"])
        st["file"] = torch.empty(len(data), dtype=torch.uint8, pin_memory=True)
        st["file"].numpy()[:] = np.frombuffer(data, dtype=np.uint8)
    else:
        n = c["rows"]
        st["ex"] = _table([("k", "int64", d.ints(0, max(1, n // 2), n, "int64") * 1_000_003),
                           ("v", "int64", d.ints(0, 10**9, n, "int64")), ("p", "int32", d.ints(0, 99, n))]).export()
        st["names"] = _abi.cstr_array(["k"])
        st["offsets"] = (ctypes.c_int64 * (c["slots"] + 1))()
    return st


_GROUP_SPEC = json.dumps({
    "groupColumnNames": ["k"], "groupsHint": 0,
    "aggregates": [aggregate("SUM", "s", col("v")), aggregate("COUNT", "n"), aggregate("MAX", "m", col("q"))],
}).encode()


def _csv_schema(fields):
    """The target schema of gfpdb_csv_read: (ArrowSchema, what keeps it)."""
    kids = (_abi.ArrowSchema * len(fields))()
    ptrs = (ctypes.POINTER(_abi.ArrowSchema) * len(fields))()
    fmt = {"int32": b"i", "date32": b"tdD", "utf8": b"u"}
    noop = _abi.SCHEMA_RELEASE(lambda p: None)
    for i, (name, ty) in enumerate(fields):
        kids[i].name = name.encode()
        kids[i].format = fmt[ty] if ty in fmt else b"d:" + ty[8:-1].replace(" ", "").encode()
        kids[i].release = noop
        ptrs[i] = ctypes.pointer(kids[i])
    s = _abi.ArrowSchema()
    s.format, s.n_children, s.release = b"+s", len(fields), noop
    s.children = ctypes.cast(ptrs, ctypes.POINTER(ctypes.POINTER(_abi.ArrowSchema)))
    return s, (kids, ptrs, noop)


def _fill_cube(t, shape, keys, values):
    """Group rows into dense cubes, one per aggregate, 0 where no group is."""
    at = np.ravel_multi_index([t[k] for k in keys], shape)
    out = {}
    for v in values:
        cube = np.zeros(shape, dtype=np.int64)
        cube.reshape(-1)[at] = t[v]
        out[v] = cube
    return out


def _placed(r, at, n):
    """A result's columns at the places its column `at` names, 0 elsewhere."""
    at = r.pop(at).long()
    return {name: torch.zeros(n, dtype=v.dtype, device=DEV).scatter_(0, at, v) for name, v in r.items()}


def run(st):
    c, L = st["case"], _abi.lib()
    kind = c["kind"]
    if kind == "batch":
        t = st["run"].execute().table
        return _fill_cube(t, (c["queries"],) + CUBE_STAR, ("query_id", "d2_g", "d4_g"), STAR_AGGS)
    if kind == "star":
        return _fill_cube(st["run"].execute().table, CUBE_STAR, ("d2_g", "d4_g"), STAR_AGGS)
    if kind == "two_table":
        t = plan.execute(st["text"], st["inputs"]).table
        at = np.array([workloads.REGIONS.index(r) for r in t["region"]], dtype=np.int64)
        out = np.zeros((2, len(workloads.REGIONS)), dtype=np.int64)
        out[0, at], out[1, at] = t["revenue"], t["cnt"]
        return {"revenue": out[0], "cnt": out[1]}
    if kind == "filter":
        return _out(L.gfpdb_filter_evaluate, st["filter"].h, st["ex"].schema_ptr, st["ex"].array_ptr, st["names"], 2)
    if kind == "bloom":
        b = _Handle(L.gfpdb_bloom_free)
        _call(L.gfpdb_bloom_create, st["dim"].schema_ptr, st["batches"], 1, st["dim_key"], 1, 10, 3, ctypes.byref(b.h),
              None)
        r = _out(L.gfpdb_bloom_use, b.h, st["fact"].schema_ptr, st["fact"].array_ptr, st["fact_key"], 1)
        return _placed(r, "c_row", c["rows"])
    if kind == "join":
        j = _Handle(L.gfpdb_hashjoin_free)
        _call(L.gfpdb_hashjoin_create, ops.JOIN_TYPES[c["type"]], st["bk"], st["pk"], 1, st["c_needed"],
              len(st["needed"]), 0.5, ctypes.byref(j.h))
        _call(L.gfpdb_hashjoin_put_build, j.h, st["b"].schema_ptr, st["b"].array_ptr, None)
        _call(L.gfpdb_hashjoin_finalize_build, j.h, None)
        r = _out(L.gfpdb_hashjoin_probe, j.h, st["p"].schema_ptr, st["p"].array_ptr)
        out = _placed(r, "c_row", c["probe"])
        if c["type"] == "LEFT":  # the build rows that no probe row found
            rest = _out(L.gfpdb_hashjoin_finish, j.h, st["p"].schema_ptr)
            out["rest"] = _placed({k: rest[k] for k in ("b_row", "b_1")}, "b_row", c["build"])
        return out
    if kind == "group":
        g = _Handle(L.gfpdb_group_free)
        _call(L.gfpdb_group_create, st["spec"], ctypes.byref(g.h))
        _call(L.gfpdb_group_update, g.h, st["ex"].schema_ptr, st["ex"].array_ptr, None)
        r = _out(L.gfpdb_group_finalize, g.h)
        r["at"] = r.pop("k") * KEY_INVERSE - 1  # the key's number in the program's own table
        return _placed(r, "at", c["keys"])
    if kind == "csv":
        return _out(L.gfpdb_csv_read, st["text"].data_ptr(), st["text"].numel(), _abi.ARROW_DEVICE_CUDA, b"|", 0,
                    ctypes.byref(st["schema"]), None, -1)
    if kind == "parquet":
        return _out(L.gfpdb_parquet_read, st["file"].data_ptr(), st["file"].numel(), None, -1, 0, -1)
    s, a = new_output()
    _call(L.gfpdb_shuffle, st["ex"].schema_ptr, st["ex"].array_ptr, st["names"], 1, c["slots"], ctypes.byref(s),
          ctypes.byref(a), st["offsets"], None)
    return _taken(s, a) | {"offsets": np.array(st["offsets"], dtype=np.int64)}


def work(case):
    c = case
    kind = c["kind"]
    if kind == "batch":  # every foreign key once, the dimensions, the groups
        n = 16 * sum(_part_sizes(c)) + 12 * sum(workloads.STAR_DIM_ROWS) + c["queries"] * 175 * 36
    elif kind == "star":  # the first probe's key, the dimensions, the groups
        n = 4 * c["rows"] + 12 * sum(workloads.STAR_DIM_ROWS) + 175 * 32
    elif kind == "two_table":
        n = 4 * c["rows"] + 0.2 * 12 * c["rows"] + 20 * c["dim_rows"] + 5 * 24
    elif kind == "filter":
        n = 12 * c["rows"] + 24 * c["rows"] * c["percent"] / 100
    elif kind == "bloom":  # keys, and the kept tenth's columns read and written
        n = 8 * c["keys"] + 8 * c["rows"] + 0.1 * c["rows"] * 48
    elif kind == "join":
        w = 4 if c["key"] == "int32" else 8
        hits = 0.5 * c["probe"]
        n = (w + 12) * c["build"] + (w + 12) * c["probe"] + 24 * hits
    elif kind == "group":
        n = 20 * c["rows"] + 28 * min(c["keys"], c["rows"])
    elif kind == "csv":
        n = c["rows"] * (241 + 4 * 4 + 4 * 8 + 2 * 4 + 6 * 29)
    elif kind == "parquet":
        n = c["rows"] * (18.5 + 32)
    else:
        n = c["rows"] * 40
    return {"bytes": n, "flops": 0}


# ------------------------------------------------------- 64-bit known answers


def _star_exact(tabs, parts, keep):
    """The cubes of one star query: keep(i, f) selects dimension i's rows by
    their filter column."""
    shape = CUBE_STAR
    cubes = torch.zeros(3, shape[0] * shape[1], dtype=torch.int64, device=DEV)
    masks = [keep(i, tabs[f"d{i + 1}"].tensors[1][0]) for i in range(4)]
    g2, g4 = tabs["d2"].tensors[2][0].long(), tabs["d4"].tensors[2][0].long()
    for p in parts:
        fk = [tabs[p].tensors[i][0].long() - 1 for i in range(4)]
        hit = torch.nonzero(masks[0][fk[0]] & masks[1][fk[1]] & masks[2][fk[2]] & masks[3][fk[3]]).reshape(-1)
        at = g2[fk[1][hit]] * shape[1] + g4[fk[3][hit]]
        qty, price, disc = (tabs[p].tensors[k][0][hit].long() for k in (4, 5, 6))
        for cube, v in zip(cubes, (price * qty, price * disc, torch.ones_like(at))):
            cube.scatter_add_(0, at, v)
    return {n: cubes[k].reshape(shape).cpu().numpy() for k, n in enumerate(STAR_AGGS)}


def exact(case, seed):
    c = case
    if c["kind"] not in ("batch", "star", "two_table", "group"):
        return None  # rows that are moved or parsed, not computed
    st = prepare(c, seed)
    if c["kind"] == "group":
        k, v, q = (x[0] for x in st["t"].tensors)
        at = k * KEY_INVERSE - 1
        zero = torch.zeros(c["keys"], dtype=torch.int64, device=DEV)
        return {"s": zero.scatter_add(0, at, v), "n": zero.scatter_add(0, at, torch.ones_like(v)),
                "m": zero.scatter_reduce(0, at, q.long(), "amax")}
    tabs = st["tables"]
    if c["kind"] == "star":
        return _star_exact(tabs, ["fact"], lambda i, f: f == workloads.STAR_DEFAULT_CONSTS[i])
    if c["kind"] == "batch":
        parts = [f"p{i}" for i in range(c["parts"])]
        each = [_star_exact(tabs, parts, lambda i, f, q=q: (f >= q[i][0]) & (f <= q[i][1])) for q in st["queries"]]
        return {n: np.stack([e[n] for e in each]) for n in STAR_AGGS}
    fk, qty, price = (x[0].long() for x in tabs["fact"].tensors)
    hit = tabs["dim"].tensors[1][0][fk - 1] < 5
    at = st["region"][fk - 1][hit]
    out = torch.zeros(2, len(workloads.REGIONS), dtype=torch.int64, device=DEV)
    out[0].scatter_add_(0, at, (price * qty)[hit])
    out[1].scatter_add_(0, at, torch.ones_like(at))
    return {"revenue": out[0].cpu().numpy(), "cnt": out[1].cpu().numpy()}
