"""Prefix sums whose total passes 2^31 are refused before anything is stored by
their offsets, also where a tile's own sum passes 2^31 or is a multiple of 2^32:
a join that repeats one long string over many rows."""

import numpy as np
import pytest

from flexpushdowndb_gb300 import _abi, ops
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

pytestmark = pytest.mark.gpu


# 2^19 rows and more are summed in tiles of 8,192 values, fewer in tiles of 2,048
@pytest.mark.parametrize("rows,length", [(1 << 19, 1 << 19), ((1 << 19) + 5, 300_000), (1 << 19, 262_144),
                                         ((1 << 19) - 1, 1 << 21), (4096, (1 << 20) + 1), (1 << 19, 4096)])
def test_oversized_total_is_refused(gpu, rows, length):
    build = Table([Column("bk", "int32", [7]), Column("bs", "utf8", ["x" * length])])
    probe = DeviceTable.from_host(Table([Column("pk", "int32", np.full(rows, 7))]))
    j = ops.HashJoin("bk", "pk", ["bs"])
    j.put_build(DeviceTable.from_host(build))
    j.finalize_build()
    with pytest.raises(_abi.GfpdbError) as e:
        j.probe(probe)
    assert e.value.code == _abi.GFPDB_EUNSUPPORTED and "2 GiB" in e.value.message
    few = j.probe(DeviceTable.from_host(Table([Column("pk", "int32", [7, 8])])))  # the library goes on as before
    assert few["bs"] == ["x" * length]
