"""The per-column kernel's accesses to an input's values (csrc/vo_column.cu) compiled for the host, at segments up to the
largest (2^31 - 1 of them): the arrays are windows of ones that are never made, so that an index out of range ends the
program. And the largest input of the patch kernel (csrc/vo_slots.h), whose entries keep such indexes signed."""
from __future__ import annotations

import os
import re
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "voroffset_gb300", "csrc")

MAIN = r"""
#include <cstdint>
#include <cstdlib>
#define __device__
#define __forceinline__ inline
struct float2 { float x, y; };
struct ColumnArgs { const double *H64, *zd; const float *zf; int W; };
static double __dadd_rn(double a, double b) { return a + b; }
static double __dsub_rn(double a, double b) { return a - b; }
#include "vo_slots.h"
@SOURCE@
// the first elements of an array of which w holds those from `first` on
template <typename T>
static const T *window(const T *w, int64_t first) {
  return reinterpret_cast<const T *>(reinterpret_cast<uintptr_t>(w) - (uintptr_t)(first * (int64_t)sizeof(T)));
}
int main(int, char **argv) {
  const int first = atoi(argv[1]), n = 8;
  if (first + (int64_t)n - 1 <= vo::kPatchSegments - 1) {  // what patches take fits a signed index
    const int64_t most = 2 * (vo::kPatchSegments - 1) + 1;
    if (most != (int32_t)most) return 2;
  }
  double z[2 * n];
  float f[2 * n];
  for (int i = 0; i < 2 * n; ++i) z[i] = 10.0 * i, f[i] = (float)i;
  const double H[1] = {3.0};
  const ColumnArgs A{H, window(z, 2 * (int64_t)first), window(f, 2 * (int64_t)first), 1};
  for (int i = 0; i < n; ++i) {
    const int k = first + i;
    const double lo = exact_val(A, @LO@, 0, false), hi = exact_val(A, @HI@, 0, true);
    if (lo != z[2 * i] - 3.0 || hi != z[2 * i + 1] + 3.0) return 1;
    const float2 c = copies_at(A.zf, k);
    if (c.x != f[2 * i] || c.y != f[2 * i + 1]) return 1;
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    src = open(os.path.join(CSRC, "vo_column.cu")).read()
    body = "".join(re.search(r"^__device__ __forceinline__ \w+ " + f + r"\(.*?}\n", src, re.S | re.M).group(0)
                   for f in ("value_index", "value_at", "copies_at", "exact_val"))
    lo, hi = re.search(r"const int il = ([^;]*?), ih = ([^;]*);", src).groups()
    d = tmp_path_factory.mktemp("index")
    (d / "main.cpp").write_text(MAIN.replace("@SOURCE@", body).replace("@LO@", lo).replace("@HI@", hi))
    # -fwrapv: 32-bit overflow as on the device
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("first", [0, 1000, (1 << 30) - 8, (1 << 30) - 4, 1 << 30, 2147483647 - 8])
def test_values_of_the_largest_inputs(program, first):
    assert subprocess.run([program, str(first)], timeout=60).returncode == 0
