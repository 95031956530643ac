"""The growth of H over one lattice step inwards (build_tables in csrc/vo_api.cu, compiled for the host): never above
the true growth of the FP64 tables, and increasing with both distances, so that the growth at a patch's nearest column
bounds that at its others; and the neighbour widths' rule with it, in a model of k_widths: a union from which the
segments held by a neighbour's candidate are left out is the same union, bit for bit."""
from __future__ import annotations

import math
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT, ogrid

CSRC = os.path.join(ROOT, "voroffset_gb300", "csrc")

MAIN = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "voroffset_gpu.h"
@SOURCE@
static double half_value(int bits) {  // of a non-negative FP16
  const int e = bits >> 10, m = bits & 1023;
  return e ? std::ldexp(1024 + m, e - 25) : std::ldexp(m, -24);
}
int main(int, char **argv) {
  Tables t;
  const double R = atof(argv[1]);
  const int rc = build_tables(R, 64, t);
  if (rc) return rc == VO_ERADIUS ? 77 : 1;
  auto H = [&](int d, int a) { return t.H[(size_t)d * t.W + a]; };
  auto grow = [&](int d, int a, bool y) {
    const unsigned g = (unsigned)t.Dx[t.Dy + 1 + (size_t)d * t.W + a];
    return (int)(short)(y ? g >> 16 : g & 0xffff);
  };
  for (int d = 0; d <= t.Dy; ++d)
    for (int a = 0; a <= t.Dx[d]; ++a)
      for (int y = 0; y < 2; ++y) {
        const int g = grow(d, a, y);
        if ((y ? d : a) == 0) {
          if (g >= 0) return printf("a growth at distance 0\n"), 2;
          continue;
        }
        if (g >= 0 && half_value(g) > (y ? H(d - 1, a) : H(d, a - 1)) - H(d, a)) return printf("%d %d above the true growth\n", d, a), 3;
        if (a + 1 <= t.Dx[d] && grow(d, a + 1, y) < g) return printf("%d %d decreases with a\n", d, a), 4;
        if (d + 1 <= t.Dy && a <= t.Dx[d + 1] && grow(d + 1, a, y) < g) return printf("%d %d decreases with d\n", d, a), 5;
        if (getenv("DUMP")) printf("%d %d %d %d\n", d, a, y, g);
      }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    header = open(os.path.join(CSRC, "vo_internal.cuh")).read()
    api = open(os.path.join(CSRC, "vo_api.cu")).read()
    parts = [re.search(r"constexpr int kPatchX = .*;", header).group(0), re.search(r"struct Tables \{.*?\n\};", header, re.S).group(0),
             re.search(r"int build_tables\(double R, int kmax, Tables &t\) \{.*?\n\}\n", api, re.S).group(0)]
    d = tmp_path_factory.mktemp("tables")
    (d / "main.cpp").write_text(MAIN.replace("@SOURCE@", "\n".join(parts)))
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT}/include", str(d / "main.cpp"), "-o", str(d / "main")],
                   check=True)
    return str(d / "main")


RADII = [0.0, 0.3, 1.0, 1.5, 2.0, 2.0000001, 4.75, 5.0, 7.07, 8.5, 13.0, 13.5, 25.0, 32.0, 32.3, 64.0, 65.0, 100.1, 127.99, 169.0,
         254.5, 255.0]


@pytest.mark.parametrize("r", RADII)
def test_growths(program, r):
    p = subprocess.run([program, repr(r)], capture_output=True, text=True)
    assert p.returncode in (0, 77), p.stdout


def trunc32(v):
    f = np.float32(v)
    return f if abs(float(f)) <= abs(v) else np.nextafter(f, np.float32(0))


def width(own, segs):
    """k_widths: bits of the width towards a neighbour with those segments."""
    lo, hi = trunc32(own[0]), trunc32(own[1])
    best = np.float32(np.inf)
    j = 0
    while j < len(segs) and trunc32(segs[j][1]) < lo:
        j += 1
    for s in segs[j:j + 2]:
        a, b = trunc32(s[0]), trunc32(s[1])
        e = np.float32(2.0 ** -21) * (abs(a) + abs(b) + abs(lo) + abs(hi)) + np.float32(1e-30)
        best = min(best, max(max(a - lo, hi - b), np.float32(0)) + e)
    h = np.float16(best)
    if float(h) < float(best):
        h = np.nextafter(h, np.float16(np.inf))
    return min(0xfff, (int(h.view(np.uint16)) + 7) >> 3)


@pytest.mark.parametrize("r,seed", [(2.0, 1), (4.75, 2), (7.07, 3)])
def test_held_segments_change_nothing(program, vo, oracle, r, seed):
    g, offs, z = vo.synth_volume(vo.SynthSpec(22, ny=19, n_spheres=14, s_rmin=2, s_rmax=8, n_cyl=2, seed=seed))
    out = subprocess.run([program, repr(r)], capture_output=True, text=True, env={**os.environ, "DUMP": "1"})
    assert out.returncode == 0
    grow = {tuple(map(int, t.split()[:3])): int(t.split()[3]) for t in out.stdout.split("\n") if t}
    nx, ny = g.nx, g.ny
    cols = [z[2 * offs[c]:2 * offs[c + 1]].reshape(-1, 2) for c in range(nx * ny)]
    near = lambda x, y: cols[x + nx * y] if 0 <= x < nx and 0 <= y < ny else np.zeros((0, 2))
    w = [[[width(s, near(c % nx + dx, c // nx + dy)) for dx, dy in ((-1, 0), (1, 0), (0, -1), (0, 1))] for s in cols[c]]
         for c in range(nx * ny)]
    wo, wz = oracle.morph(ogrid(oracle, g), offs, z, r, "dilation")
    R = [r if d == 0 else math.sqrt(r * r - d * d) for d in range(int(r) + 1)]
    kept = total = 0
    for c in range(nx * ny):
        x, y = c % nx, c // nx
        cand = []
        for d in range(int(r) + 1):
            for a in range(int(math.floor(R[d])) + 1):
                h = math.sqrt(R[d] * R[d] - a * a)
                for sx in {x - a, x + a}:
                    for sy in {y - d, y + d}:
                        if not (0 <= sx < nx and 0 <= sy < ny):
                            continue
                        for i, s in enumerate(cols[sx + nx * sy]):
                            total += 1
                            wx, wy = w[sx + nx * sy][i][1 if sx < x else 0], w[sx + nx * sy][i][3 if sy < y else 2]
                            if (a and wx << 3 <= grow[(d, a, 0)]) or (d and wy << 3 <= grow[(d, a, 1)]):
                                continue
                            kept += 1
                            cand.append((s[0] - h, s[1] + h))
        cand.sort()
        union = []
        for lo, hi in cand:
            if union and lo <= union[-1][1]:
                union[-1][1] = max(union[-1][1], hi)
            else:
                union.append([lo, hi])
        assert np.array_equal(np.array(union).reshape(-1), wz[2 * wo[c]:2 * wo[c + 1]]), c
    assert kept < 0.8 * total
