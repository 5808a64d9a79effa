"""Host-side checks of the resident iterations' preparation: the cut of a
plan's tiles into pieces covers every element once, keeps to its limits and
balances the SMs, and the bit conversions between float and double that
replace the GPU's conversion instructions are exact (a C++ program built from
the package's own sources)."""

from __future__ import annotations

import pathlib
import re
import subprocess

ROOT = pathlib.Path(__file__).resolve().parent.parent
CSRC = ROOT / "apple_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include "agb_internal.h"
using namespace agb;

static uint32_t __float_as_uint(float x) { uint32_t b; memcpy(&b, &x, 4); return b; }
static float __uint_as_float(uint32_t b) { float x; memcpy(&x, &b, 4); return x; }
static double __hiloint2double(int h, int l) {
  uint64_t v = (uint64_t)(uint32_t)h << 32 | (uint32_t)l; double d; memcpy(&d, &v, 8); return d;
}
static uint64_t bits(double d) { uint64_t v; memcpy(&v, &d, 8); return v; }
static int __double2hiint(double d) { return (int)(bits(d) >> 32); }
static int __double2loint(double d) { return (int)bits(d); }
CONVERSIONS

static int split(int tiles, int groups, std::mt19937& rng) {
  TilePlan p, q;
  p.tile_estart.assign(1, 0); p.tile_vstart.assign(1, 0); p.tile_gstart.assign(1, 0);
  for (int t = 0; t < tiles; ++t) {
    const int g = 1 + (int)(rng() % (2 * groups)), nv = 4 + (int)(rng() % 250);
    for (int k = 0; k < g; ++k) { p.group_estart.push_back(p.n_cells); p.n_cells += 1 + (int)(rng() % 32); }
    for (int k = 0; k < nv; ++k) p.tv_vid.push_back((int)rng() % 1000);
    p.tile_estart.push_back(p.n_cells);
    p.tile_vstart.push_back((int)p.tv_vid.size());
    p.tile_gstart.push_back((int)p.group_estart.size());
  }
  p.group_estart.push_back(p.n_cells);
  p.n_tiles = tiles; p.n_tv = (int)p.tv_vid.size();
  split_tiles(p, 152, 2, &q);
  if (q.n_tiles < tiles || q.n_tiles > 304 || (int)q.tile_gstart.size() != q.n_tiles + 1) return 1;
  int t = 0;
  for (int k = 0; k < q.n_tiles; ++k) {
    while (q.tile_gstart[k] >= p.tile_gstart[t + 1]) ++t;
    const int a = q.tile_gstart[k], b = q.tile_gstart[k + 1];
    if (b <= a || b > p.tile_gstart[t + 1]) return 2;                      // inside one tile
    if (q.tile_estart[k] != p.group_estart[a] || q.tile_estart[k + 1] != p.group_estart[b]) return 3;
    const int n = q.tile_vstart[k + 1] - q.tile_vstart[k];
    if (n != p.tile_vstart[t + 1] - p.tile_vstart[t]) return 4;
    if (memcmp(&q.tv_vid[q.tile_vstart[k]], &p.tv_vid[p.tile_vstart[t]], n * sizeof(int32_t))) return 5;
    const bool cut = b - a < p.tile_gstart[t + 1] - p.tile_gstart[t];
    if (cut && b - a < 8) return 6;
    if (cut && tiles > 152 && k < 152) return 7;                           // the first 152 stay whole
  }
  if (q.tile_gstart.back() != p.tile_gstart.back()) return 8;
  return 0;
}

int main() {
  std::mt19937 rng(1);
  for (int tiles : {1, 2, 8, 75, 76, 77, 151, 152, 153, 154, 204, 300, 303, 304})
    for (int groups : {1, 4, 11, 30})
      if (int e = split(tiles, groups, rng)) { printf("split %d %d: %d\n", tiles, groups, e); return 1; }
  std::mt19937_64 g(2);
  for (uint64_t i = 0; i < 20000000; ++i) {
    const float f = __uint_as_float((uint32_t)g());
    if (f == f && bits(widen(f)) != bits((double)f)) { printf("widen %a\n", f); return 2; }
    uint64_t v = g();
    if (i & 1) v = (v & 0x800fffffffffffffull) | (uint64_t)(880 + g() % 290) << 52;  // around float's range
    if ((i & 7) == 3) v &= ~0x1fffffffull;
    if ((i & 7) == 5) v = (v & ~0x1fffffffull) | 0x10000000ull;                       // ties
    if ((i & 15) == 7) v |= 0x000fffffe0000000ull;                                    // carries
    double d; memcpy(&d, &v, 8);
    if (d == d && __float_as_uint(narrow(d)) != __float_as_uint((float)d)) { printf("narrow %a\n", d); return 3; }
  }
  for (double d : {0.0, -0.0, 1e-320, 1e300, -1e300, 3.4028235677973366e38})
    if (__float_as_uint(narrow(d)) != __float_as_uint((float)d)) return 4;
  return 0;
}
"""


def test_split_tiles_and_conversions(tmp_path):
    src = (CSRC / "reduce.cuh").read_text()
    body = re.search(r"__device__ __forceinline__ double widen.*?\n}\n__device__ __forceinline__ float narrow.*?\n}\n",
                     src, re.S).group(0).replace("__device__ __forceinline__", "static")
    cpp = tmp_path / "check.cpp"
    cpp.write_text(PROGRAM.replace("CONVERSIONS", body))
    exe = tmp_path / "check"
    cuda = pathlib.Path("/usr/local/cuda/include")
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", f"-I{cuda}", str(cpp), str(CSRC / "prep.cpp"), "-o",
                    str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
