"""Hash join tables probed by four-slot groups, against sorted numpy joins:
probe batches around a warp's step, builds that fill groups past their end
(high load factors, few distinct keys repeated many times, keys that come back
in later groups), 32- and 64-bit keys, every join type, and a build side kept
to the columns the join needs."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import GfpdbError, ops
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu


def tables(nb, n, distinct, ty, seed):
    rng = np.random.default_rng(seed)
    scale = 1 if ty == "int32" else (1 << 33) + 1
    b = Table([Column("bk", ty, rng.integers(0, distinct, nb) * scale), Column("bv", "int64", np.arange(nb)),
               Column("unused", "int64", np.zeros(nb))])
    p = Table([Column("pk", ty, rng.integers(0, 2 * distinct, n) * scale), Column("pv", "int32", np.arange(n))])
    return b, p


def pairs(b, p):
    """(probe row, build row) of every match, sorted."""
    order = np.argsort(b["bk"], kind="stable")
    keys = b["bk"][order]
    lo, hi = np.searchsorted(keys, p["pk"], "left"), np.searchsorted(keys, p["pk"], "right")
    pr = np.repeat(np.arange(p.num_rows), hi - lo)
    at = np.repeat(lo, hi - lo) + (np.arange(len(pr)) - np.repeat(np.cumsum(hi - lo) - (hi - lo), hi - lo))
    return sorted(zip(pr.tolist(), order[at].tolist()))


def join(b, p, kind="INNER", lf=0.5, batches=1):
    j = ops.HashJoin("bk", "pk", ["pv", "bv"], load_factor=lf, join_type=kind)
    step = (b.num_rows + batches - 1) // batches
    for i in range(0, max(b.num_rows, 1), max(step, 1)):
        j.put_build(DeviceTable.from_host(b.slice(i, min(b.num_rows, i + step))))
    j.finalize_build()
    out = j.probe(DeviceTable.from_host(p))
    return out, (j.finish() if kind in ("LEFT", "FULL", "LEFT_SEMI") else None)


@pytest.mark.parametrize("ty", ["int32", "int64"])
@pytest.mark.parametrize("n", [1, 31, 63, 64, 65, 127, 128, 2047, 70_001])
@pytest.mark.parametrize("nb,distinct,lf", [(1, 1, 0.5), (5, 3, 0.9), (57, 57, 0.9), (900, 1000, 0.9), (40_000, 30_000, 0.9),
                                            (40_000, 50_000, 0.3)])
def test_inner(gpu, ty, n, nb, distinct, lf):
    b, p = tables(nb, n, distinct, ty, n + nb)
    out, _ = join(b, p, lf=lf, batches=2 if nb > 50 else 1)
    assert sorted(zip(out["pv"].tolist(), out["bv"].tolist())) == pairs(b, p)


@pytest.mark.parametrize("n", [1, 64, 300])
def test_long_runs_of_one_key(gpu, n):
    """One key on hundreds of build rows: its run covers many groups, and a
    probe row emits hundreds of matches."""
    b, p = tables(700, n, 2, "int32", n)
    out, _ = join(b, p)
    assert sorted(zip(out["pv"].tolist(), out["bv"].tolist())) == pairs(b, p)


@pytest.mark.parametrize("kind", ["LEFT", "RIGHT", "FULL", "LEFT_SEMI", "RIGHT_SEMI"])
@pytest.mark.parametrize("ty", ["int32", "int64"])
def test_other_kinds(gpu, kind, ty):
    b, p = tables(3001, 5003, 2500, ty, 7)
    m = pairs(b, p)
    out, rest = join(b, p, kind, lf=0.9)
    hit_p, hit_b = {x for x, _ in m}, {y for _, y in m}
    if kind == "LEFT_SEMI":
        assert sorted(rest["bv"].tolist()) == sorted(hit_b)
        return
    if kind == "RIGHT_SEMI":
        assert sorted(out["pv"].tolist()) == sorted(hit_p)
        return
    rows = out.rows()
    want = m + ([(x, None) for x in range(p.num_rows) if x not in hit_p] if kind in ("RIGHT", "FULL") else [])
    assert sorted(rows, key=str) == sorted(want, key=str)
    if kind in ("LEFT", "FULL"):
        assert sorted(rest["bv"].tolist()) == [y for y in range(b.num_rows) if y not in hit_b]


def test_columns_not_needed_still_count(gpu):
    """A build column that the join drops is still checked: batches must
    agree on it."""
    b, _ = tables(10, 1, 5, "int32", 1)
    other = Table([c if c.name != "unused" else Column("unused", "int32", np.zeros(10)) for c in b.columns])
    j = ops.HashJoin("bk", "pk", ["pv", "bv"])
    j.put_build(DeviceTable.from_host(b))
    j.put_build(DeviceTable.from_host(other))
    with pytest.raises(GfpdbError, match="schema mismatch on column 'unused'"):
        j.finalize_build()
    j = ops.HashJoin("bk", "pk", ["pv", "bv"])
    j.put_build(b)  # a host batch and a device batch of the same schema
    j.put_build(DeviceTable.from_host(b))
    j.finalize_build()
    assert j.info()["build_rows"] == 20
