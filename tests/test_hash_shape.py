"""The hash scan's shared-memory table by plan width and capacity (ws_shape.h): wide plans keep a table, copies of the
first keys' accumulators never displace slots, and everything fits an SM."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAIN = r"""
#include <cstdio>
#include "ws_shape.h"
int main() {
  for (int compiled = 0; compiled < 2; ++compiled)
    for (int sums = 1; sums <= 40; ++sums)
      for (int keys = 1; keys <= 4; ++keys)
        for (int resident = 1; resident <= 4; ++resident)
          for (int log = 1; log <= 24; ++log) {
            const size_t acc = compiled ? 4 + 12 * (size_t)sums : 16 + 16 * (size_t)sums;
            const size_t slot = 9 + acc + (keys > 1 ? 8 * (size_t)keys : 0);
            const ws::HashTable t = ws::hashTable((int64_t)1 << log, slot, acc, 16, 8, resident, 0, compiled);
            printf("%d %d %d %d %d %zu %zu %zu %d %zu %zu\n", compiled, sums, keys, resident, log, acc, slot, t.slots, t.copies,
                   t.bytes, t.spill);
          }
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    src = d / "shape.cpp"
    src.write_text(MAIN)
    exe = str(d / "shape")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "warpstore_b200", "csrc"), str(src), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [tuple(int(x) for x in line.split()) for line in out.splitlines()]


def test_wide_plans_keep_a_table(shapes):
    for compiled, sums, keys, resident, log, acc, slot, slots, copies, nbytes, spill in shapes:
        what = (compiled, sums, keys, resident, log)
        if 64 * slot <= 48 * 1024:
            assert slots >= 64, what
        assert slots & (slots - 1) == 0 and slots <= 4096, what


def test_copies_take_only_what_slots_leave(shapes):
    for compiled, sums, keys, resident, log, acc, slot, slots, copies, nbytes, spill in shapes:
        what = (compiled, sums, keys, resident, log)
        assert nbytes == slots * slot + (16 * copies * acc if copies > 1 else 0), what
        assert copies == 1 or nbytes <= max(56 * 1024, 226 * 1024 // max(resident - 1, 1) - 1024 - 8 * 1024), what
        assert nbytes + spill + 1024 <= 226 * 1024, what


def test_narrow_plans_keep_their_ctas(shapes):
    """COUNT and up to eight SUMs at four resident CTAs: the table and its buffer leave room for three."""
    for compiled, sums, keys, resident, log, acc, slot, slots, copies, nbytes, spill in shapes:
        if compiled and sums <= 8 and resident == 4:
            assert 3 * (nbytes + spill + 1024) <= 227 * 1024, (sums, keys, log)
