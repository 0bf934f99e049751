"""Device-to-device copies whose ends are aligned alike or not: build batches of
device columns that begin anywhere in their buffers, and the concatenation of
parts of odd sizes, so that every offset modulo 16 occurs, by a join that brings
each build row back."""

import numpy as np
import pytest
import torch

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu

TORCH = {"int32": torch.int32, "int64": torch.int64, "date32": torch.int32, "float64": torch.float64}


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("sizes", [[1], [2, 3], [7, 9, 11, 13], [31, 33, 64, 65], [1001, 5, 70_001], [4097] * 70])
def test_parts(gpu, shift, sizes):
    rng = np.random.default_rng(shift + sum(sizes))
    n = sum(sizes)
    values = {"bk": ("int32", rng.permutation(n)), "b": ("int64", rng.integers(-(1 << 62), 1 << 62, n)),
              "c": ("int32", rng.integers(0, 1 << 30, n)), "d": ("date32", rng.integers(0, 20_000, n)),
              "e": ("float64", rng.normal(0, 1, n))}
    j = ops.HashJoin("bk", "pk")
    at, held = 0, []
    for m in sizes:
        tensors = []
        for ty, v in values.values():
            buf = torch.empty(m + 4, dtype=TORCH[ty], device="cuda")
            buf[shift : shift + m] = torch.from_numpy(np.asarray(v[at : at + m])).to(TORCH[ty])
            tensors.append([buf[shift : shift + m]])
        held.append(DeviceTable(list(values), [ty for ty, _ in values.values()], tensors, m))
        j.put_build(held[-1])
        at += m
    j.finalize_build()
    got = j.probe(DeviceTable.from_host(Table([Column("pk", "int32", np.arange(n))])))
    order = np.argsort(got["pk"], kind="stable")
    assert np.array_equal(np.asarray(got["pk"])[order], np.arange(n))
    back = np.argsort(values["bk"][1])
    for name in "bcde":
        want = values[name][1][back]
        assert np.array_equal(np.asarray(got[name])[order], want.astype(np.asarray(got[name]).dtype)), name
