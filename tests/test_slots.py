"""The slot layout of a single dilation (csrc/vo_slots.h) on grids up to the largest (2^26 columns): its index
range, and that every result of up to 2^31 - 1 segments gets its slots within three runs, whatever its columns' counts."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "vo_slots.h"
using namespace vo;
// columns with counts[i] intervals in `part[i]` of the columns: the spill space that a run asks for
int main(int, char **argv) {
  const int64_t ncols = atoll(argv[1]);
  const double mean = atof(argv[2]);
  const int64_t many = atoll(argv[3]), few = atoll(argv[4]);  // intervals of the columns that have many, of the others
  const int64_t rich = atoll(argv[5]);                        // how many have many
  if (rich * many + (ncols - rich) * few > kSegmentsMost) return 3;
  SlotLayout s = slots_first(ncols, mean);
  if (atoi(argv[6])) slots_many(ncols, s);
  for (int run = 0; run < 3; ++run) {
    if (s.cap < 1 || s.cap * ncols + s.spill > kSlotMost) return 4;
    const int64_t need = (many > s.cap ? rich * many : 0) + (few > s.cap ? (ncols - rich) * few : 0);
    if (need <= s.spill) return 0;
    if (run == 2 || !slots_next(ncols, need, s)) return 5;
  }
  return 6;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("slots")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT}/voroffset_gb300/csrc", str(d / "main.cpp"), "-o", str(d / "main")],
                   check=True)
    return str(d / "main")


LARGEST = 1 << 26
CASES = [(1, 1.0, 500, 0, 1), (4096, 3.0, 8000, 1, 4096), (LARGEST, 1.0, 31, 31, LARGEST), (LARGEST, 12.0, 49, 15, 30_000_000),
         (LARGEST, 12.0, 49, 0, 43_000_000), (LARGEST, 25.0, 57, 20, 20_000_000), (LARGEST, 2.0, 8192, 0, 262_000),
         (LARGEST - 1, 30.0, 65, 0, 33_000_000), (LARGEST, 6.5, 33, 31, 1_000_000), (50_000_000, 40.0, 60, 42, 600_000)]


# `large`: from the layout for inputs most of whose columns have large unions
@pytest.mark.parametrize("large", [0, 1])
@pytest.mark.parametrize("ncols,mean,many,few,rich", CASES)
def test_any_result_gets_its_slots(program, ncols, mean, many, few, rich, large):
    r = subprocess.run([program, str(ncols), str(mean), str(many), str(few), str(rich), str(large)])
    assert r.returncode == 0
