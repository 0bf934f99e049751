"""The dynamic shared-memory limit of a kernel belongs to the kernel on a device,
so calls from several threads only ever raise it: the bookkeeping on the CPU
against a stand-in for the runtime's call, and shuffles of both tile sizes and
several slot counts from two threads on the GPU."""

import subprocess
import threading
from pathlib import Path

import numpy as np
import pytest

from flexpushdowndb_gb300 import ops
from flexpushdowndb_gb300.tupleset import Column, DeviceTable, Table

HOST = Path(__file__).resolve().parent.parent / "flexpushdowndb_gb300" / "csrc" / "host"

PROGRAM = r"""
#include "shared_limits.h"
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>
int main() {
  gfpdb::SharedLimits limits;
  int kernels[3];
  int now[2][3] = {};  // the runtime's own values, by device and kernel
  std::atomic<int> lowered{0}, short_of{0}, calls{0};
  auto ask = [&](int device, int k, int bytes) {
    limits.raise(device, &kernels[k], bytes, [&](int b) {
      if (b < now[device][k]) ++lowered;
      now[device][k] = b;
      ++calls;
    });
  };
  std::vector<std::thread> ts;
  for (int t = 0; t < 4; ++t)
    ts.emplace_back([&, t] {
      for (int i = 0; i < 20000; ++i) {
        const int device = (i + t) % 2, k = i % 3, bytes = 1000 + (i * 7919 + t * 104729) % 90000;
        ask(device, k, bytes);
        limits.raise(device, &kernels[k], 0, [](int) {});  // under the lock: what a launch would find
        limits.raise(device, &kernels[k], bytes, [&](int) { ++short_of; });
      }
    });
  for (auto& t : ts) t.join();
  const int before = calls;
  ask(0, 0, 5);  // less than it has
  bool threw = false;
  try {
    limits.raise(1, &kernels[2], 1 << 20, [](int) { throw std::runtime_error("refused"); });
  } catch (const std::runtime_error&) { threw = true; }
  int again = 0;
  limits.raise(1, &kernels[2], 1 << 20, [&](int b) { again = b; });  // tried again
  std::printf("%d %d %d %d %d", lowered.load(), short_of.load(), calls - before, threw ? 1 : 0, again);
}
"""


def test_limits_only_rise(tmp_path):
    src = tmp_path / "limits.cpp"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{HOST}", str(src), "-o", str(tmp_path / "limits")], check=True)
    assert subprocess.run([str(tmp_path / "limits")], capture_output=True, text=True, check=True).stdout == f"0 0 0 1 {1 << 20}"


def test_every_limit_is_kept_per_device():
    """A process may use several devices, and each has its own limits: no
    source sets one but allow_shared."""
    sources = [p for kind in ("*.cu", "*.cuh", "*.cpp", "*.h") for p in HOST.parent.rglob(kind)]
    assert len(sources) > 10
    assert [p.name for p in sources if "MaxDynamicSharedMemorySize" in p.read_text()] == ["runtime.cpp"]


@pytest.mark.gpu
@pytest.mark.parametrize("slots", [(256, 256), (1000, 300), (20, 32)])
def test_shuffles_from_two_threads(gpu, slots):
    rows = (2_000_000, 10_000)  # tiles of 16 warps and of 8
    tables = [DeviceTable.from_host(Table([Column("k", "int64", np.arange(n)), Column("v", "int32", np.arange(n))])) for n in rows]
    failed = []

    def work(i):
        try:
            for _ in range(100 if i == 0 else 400):
                _, offsets = ops.shuffle(tables[i], "k", slots[i])
                assert offsets[0] == 0 and offsets[-1] == rows[i]
        except Exception as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
