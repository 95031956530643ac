"""compact_columns (csrc/vo_internal.cuh) compiled for the host, its warp's lanes as 32 threads that meet at
every shuffle: columns of any counts against a plain copy, and offsets up to the largest that a volume may
have (2^31 - 1), where positions beyond the end no longer fit 32 bits. The output array of that case is a window
at the end of an array that is never made: a position out of range ends the program."""
from __future__ import annotations

import os
import re
import subprocess

import pytest

from conftest import ROOT

MAIN = r"""
#include <algorithm>
#include <barrier>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
using std::min;
struct double2 { double x, y; };
struct Dim { int x; };
static thread_local Dim threadIdx;
static Dim blockIdx{0}, blockDim{32};
static long long exchanged[32];
static std::barrier<> meet(32);
template <typename T>
T __shfl_sync(unsigned, T v, int from) {
  exchanged[threadIdx.x] = (long long)v;
  meet.arrive_and_wait();
  const T r = (T)exchanged[from & 31];
  meet.arrive_and_wait();
  return r;
}
@SOURCE@
int main(int argc, char **argv) {
  const int ncols = atoi(argv[1]);
  const long long first = atoll(argv[2]);
  srand(atoi(argv[3]));
  std::vector<int32_t> offs(ncols + 1);
  std::vector<std::vector<double2>> cols(ncols);
  offs[0] = (int32_t)first;
  for (int c = 0; c < ncols; ++c) {
    const int n = rand() % 4 == 0 ? 0 : rand() % 7;
    for (int k = 0; k < n; ++k) cols[c].push_back({c + 0.25 * k, c + 100.0 * k});
    offs[c + 1] = (int32_t)std::min<long long>(offs[c] + (long long)n, 2147483647LL);
  }
  if (first > 1000) offs[ncols] = 2147483647;  // up to the largest total
  while (ncols && (long long)cols[ncols - 1].size() < offs[ncols] - offs[ncols - 1]) cols[ncols - 1].push_back({7, 7});
  const long long total = offs[ncols] - first;
  std::vector<double2> out(total + 1, double2{-1, -1});
  double2 *oz = reinterpret_cast<double2 *>(reinterpret_cast<uintptr_t>(out.data()) - (uintptr_t)(16 * first));
  for (int w = 0; w < (ncols + 31) / 32; ++w) {
    blockIdx.x = w;
    std::vector<std::thread> lanes;
    for (int l = 0; l < 32; ++l)
      lanes.emplace_back([&, l] {
        threadIdx.x = l;
        vo_test::compact_columns(ncols, offs.data(), oz, [&](int c) { return (const double2 *)cols[c].data(); });
      });
    for (auto &t : lanes) t.join();
  }
  for (int c = 0; c < ncols; ++c)
    for (int k = 0; k < offs[c + 1] - offs[c]; ++k) {
      const double2 v = out[offs[c] - first + k];
      if (v.x != cols[c][k].x || v.y != cols[c][k].y) return printf("column %d\n", c), 1;
    }
  return out[total].x == -1 ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    src = open(os.path.join(ROOT, "voroffset_gb300", "csrc", "vo_internal.cuh")).read()
    body = re.search(r"template <typename Src>\n__device__ __forceinline__ void compact_columns\(.*?\n}\n", src, re.S).group(0)
    d = tmp_path_factory.mktemp("compact")
    (d / "main.cpp").write_text(MAIN.replace("@SOURCE@", "namespace vo_test {\n" + body + "}"))
    # -fwrapv: 32-bit overflow as on the device
    subprocess.run(["g++", "-std=c++20", "-O1", "-fwrapv", "-pthread", str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return str(d / "main")


# several seeds at the end of the range: how far a warp's last turn reaches beyond the end depends on the counts
@pytest.mark.parametrize("ncols,first", [(1, 0), (32, 0), (77, 5), (32, 2147483647 - 61), (32, 2147483647 - 90), (96, 2147483647 - 280)])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_compact_columns(program, ncols, first, seed):
    assert subprocess.run([program, str(ncols), str(first), str(seed)], timeout=60).returncode == 0
